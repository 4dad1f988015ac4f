"""Planned batches in several chunks (a scratch limit of one beam and of a few):
the dose and fluence gradient of the direct call, also after the fluence changes
so that the crop boxes shrink and grow, in both kernel modes, on cubes and on
voxels that are not cubes (where the bounds hold whole arrays).  No beam exceeds
a bound of its plan.

Tolerance: the same terms in another order of float atomics, 1e-5 of the
maximum, as the repository's other batch tests.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


def close(a, b):
    np.testing.assert_allclose(a, b, rtol=0, atol=1e-5 * np.abs(b).max())


@pytest.mark.parametrize("limit", [1 << 20, 48 << 20, 8 << 30])
@pytest.mark.parametrize("mode,cubes", [("exp", True), ("exp", False), ("table", True)])
def test_plan_in_chunks(mode, cubes, limit):
    import torch
    vol = inputs.head_neck_phantom(shape=(43, 38, 35), voxel_cm=0.3)
    if not cubes:
        vol.voxel = np.array([0.33, 0.27, 0.3])
        vol.start = -0.5 * (np.array([43, 38, 35]) - 1) * vol.voxel
    rng = np.random.default_rng(15)
    bs = []
    for k, (g, c) in enumerate(inputs.four_pi_angles(9, seed=6)):
        b = inputs.single_beam(fmap=(1 + k, 9 - k), beamlet_cm=0.41, gantry_deg=float(g), couch_deg=float(c),
                               coll_deg=13.0 * k, iso=(0.9 * (k % 4) - 1.513, 0.207, 1.1 * (k % 3) - 1.311))
        b.fluence = rng.uniform(0.2, 1.0, b.fluence.shape).astype(np.float32)
        bs.append(b)
    g = rng.standard_normal(vol.density.shape).astype(np.float32)
    phys = inputs.make_physics(seed=1, spacing_cm=0.3)
    with engine.Engine(0) as e, engine.Engine(0) as ref:
        for x in (e, ref):
            x.set_volume(vol)
            x.set_physics(phys, mode=mode)
        e.set_scratch_limit(limit)
        fl = torch.from_numpy(engine.concat_fluence(bs)).cuda()
        dose, grad, fg = torch.zeros(vol.nvoxels, device="cuda"), torch.from_numpy(g.ravel()).cuda(), torch.zeros_like(fl)
        plan = e.plan(bs, fl.data_ptr(), dose.data_ptr(), grad.data_ptr(), fg.data_ptr())
        chunks = plan.info()["chunks"]
        assert chunks == 9 if limit == 1 << 20 else chunks == 1 if limit == 8 << 30 else 1 < chunks < 9
        for keep in (1.0, 0.2):  # share of the beamlets that stay open
            for b in bs:
                b.fluence = (rng.uniform(0.2, 1.0, b.fluence.shape) * (rng.random(b.fluence.shape) < keep)).astype(np.float32)
                b.fluence[0, 0] = 0.7
            fl.copy_(torch.from_numpy(engine.concat_fluence(bs)))
            torch.cuda.synchronize()
            plan.launch()
            assert plan.status() == 0
            want = ref.beam_dose(bs)
            close(dose.cpu().numpy().reshape(want.shape), want)
            close(fg.cpu().numpy(), np.concatenate([f.ravel() for f in ref.beam_dose_adjoint(bs, g)]))
        plan.close()
