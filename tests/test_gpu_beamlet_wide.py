"""Columns of beamlets whose source search is split over several warps, as wide
and few ones are: the same CSR, bit for bit, from a launch per direction (a small
scratch limit, more warps to a pillar) as from one launch of all directions.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,width", [(1, 0.25), (1, 4.0), (1, 9.0), (2, 2.5), (3, 1.1), (9, 0.25)])
def test_columns_do_not_depend_on_the_split(n, width):
    vol = inputs.head_neck_phantom(shape=(43, 51, 38), voxel_cm=0.25)
    beam = inputs.single_beam(fmap=(n, n), beamlet_cm=width, gantry_deg=31.0, couch_deg=14.0, coll_deg=6.0)
    out = []
    for limit in (1 << 20, 8 << 30):
        with engine.Engine(0) as e:
            e.set_volume(vol)
            e.set_physics(inputs.make_physics(seed=4, spacing_cm=0.25), mode="table")
            e.set_scratch_limit(limit)
            out.append(e.beamlet_columns(beam))
    assert len(out[0][2]) > 0
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
