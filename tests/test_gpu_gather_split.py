"""The forward gather's three launch shapes (few, some and many blocks) on the
same beams: each beam's dose alone, among 4 and among 30.

Tolerance: a voxel sums the same terms in the same order in all three; where the
compiler fuses a multiply-add in one and not in the other, a term moves by a few
units of 2^-24: 2e-6 of the maximum.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(67, 120, 96), (131, 97, 101)])
def test_dose_of_a_beam_alone_and_among_others(shape):
    vol = inputs.head_neck_phantom(shape=shape, voxel_cm=0.25)
    rng = np.random.default_rng(3)
    bs = []
    for k, (g, c) in enumerate(inputs.four_pi_angles(30, seed=9)):
        b = inputs.single_beam(fmap=(36 + k % 3, 35 + k % 2), beamlet_cm=0.5, gantry_deg=float(g), couch_deg=float(c),
                               coll_deg=7.0 * k, iso=(0.213, -0.107, 0.311))
        b.fluence = rng.uniform(0.2, 1.0, b.fluence.shape).astype(np.float32)
        bs.append(b)
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(inputs.make_physics(seed=2, spacing_cm=0.25), mode="exp")
        d = {n: e.beam_dose(bs[:n], per_beam=True) for n in (1, 4, 30)}
    for n in (1, 4):
        for k in range(n):
            np.testing.assert_allclose(d[n][k], d[30][k], rtol=0, atol=2e-6 * np.abs(d[30][k]).max())
