"""Beamlet columns with the convolution directions in one launch and in groups
that a scratch limit forces: the dose of a voxel sums the directions in order
either way, so the columns are the same bit for bit."""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmap,beamlet", [((1, 1), 0.25), ((3, 2), 1.9), ((5, 4), 0.3)])
def test_directions_in_groups(fmap, beamlet):
    vol = inputs.head_neck_phantom(shape=(45, 38, 41), voxel_cm=0.3)
    phys = inputs.make_physics(seed=2, spacing_cm=0.3)
    beam = inputs.single_beam(fmap=fmap, beamlet_cm=beamlet, gantry_deg=28.0, couch_deg=13.0)
    out = []
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(phys, mode="table")
        for limit in (8 << 30, 1 << 20, 24 << 20):  # all 24 directions, one at a time, a few
            e.set_scratch_limit(limit)
            out.append(e.beamlet_columns(beam, 1e-4))
    assert len(out[0][3]) > 0
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
