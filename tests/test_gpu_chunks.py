"""Beams in one chunk and in chunks of one (a small scratch limit): the same
dose and fluence gradient, and a planned batch whose crop boxes shrink and grow
again with the fluence.

Tolerance: the beams' doses and the adjoint's sums are added with float atomics
in another order, a few units of 2^-24 of the largest term: rtol 1e-5 of the
maximum, as the repository's other batch tests.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


def beams(n):
    rng = np.random.default_rng(5)
    out = []
    for k, (g, c) in enumerate(inputs.four_pi_angles(n, seed=4)):
        b = inputs.single_beam(fmap=(3 + k % 4, 2 + k % 5), beamlet_cm=0.41, gantry_deg=float(g), couch_deg=float(c),
                               coll_deg=11.0 * k, iso=(0.5 * (k % 3) - 0.513, 0.207, -0.311))
        b.fluence = rng.uniform(0.2, 1.0, b.fluence.shape).astype(np.float32)
        out.append(b)
    return out


def close(a, b):
    np.testing.assert_allclose(a, b, rtol=0, atol=1e-5 * np.abs(b).max())


@pytest.mark.parametrize("mode", ["exp", "table", "walk"])
def test_chunks_of_one_beam(mode):
    vol = inputs.head_neck_phantom(shape=(43, 38, 35), voxel_cm=0.3)
    bs = beams(7)
    g = np.random.default_rng(6).standard_normal(vol.density.shape).astype(np.float32)
    out = []
    for limit in (8 << 30, 1 << 20):
        with engine.Engine(0) as e:
            e.set_volume(vol)
            e.set_physics(inputs.make_physics(seed=1, spacing_cm=0.3), mode=mode)
            e.set_scratch_limit(limit)
            out.append((e.beam_dose(bs), e.beam_dose(bs, per_beam=True), np.concatenate([f.ravel() for f in e.beam_dose_adjoint(bs, g)])))
    for a, b in zip(out[1], out[0]):
        close(a, b)


def test_plan_with_other_fluences():
    import torch
    vol = inputs.head_neck_phantom(shape=(43, 38, 35), voxel_cm=0.3)
    bs = beams(6)
    rng = np.random.default_rng(7)
    g = rng.standard_normal(vol.density.shape).astype(np.float32)
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(inputs.make_physics(seed=1, spacing_cm=0.3), mode="exp")
        fl = torch.from_numpy(engine.concat_fluence(bs)).cuda()
        dose, grad, fg = torch.zeros(vol.nvoxels, device="cuda"), torch.from_numpy(g.ravel()).cuda(), torch.zeros_like(fl)
        plan = e.plan(bs, fl.data_ptr(), dose.data_ptr(), grad.data_ptr(), fg.data_ptr())
        for keep in (0.1, 1.0, 0.5):  # share of the beamlets that stay open
            for b in bs:
                b.fluence = (rng.uniform(0.2, 1.0, b.fluence.shape) * (rng.random(b.fluence.shape) < keep)).astype(np.float32)
                b.fluence[0, 0] = 0.7
            fl.copy_(torch.from_numpy(engine.concat_fluence(bs)))
            torch.cuda.synchronize()
            plan.launch()
            assert plan.status() == 0
            ref = e.beam_dose(bs)
            close(dose.cpu().numpy().reshape(ref.shape), ref)
            close(fg.cpu().numpy(), np.concatenate([f.ravel() for f in e.beam_dose_adjoint(bs, g)]))
        plan.close()
