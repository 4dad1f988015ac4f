"""Adjoint of dose gradients that are zero almost everywhere, for which most line
tiles stay out of the cones' lists: A^T(gd + gs) - A^T gd = A^T gs, with gs one
voxel, the corners of the volume, a small box, and nothing.

Tolerance: each adjoint's float sums run in another order, 1e-5 of the maximum
as in the other batch tests, and the difference has two of them: 2e-5 of the
dense gradient's maximum.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


def sparse(kind, shape, rng):
    g = np.zeros(shape, np.float32)
    if kind == "voxel":
        g[shape[0] // 2, shape[1] // 2 + 1, shape[2] // 2] = 3.0
    elif kind == "corners":
        for c in np.ndindex(2, 2, 2):
            g[tuple(-k for k in c)] = 2.0
    elif kind == "box":
        g[20:27, 15:30, 11:18] = rng.standard_normal((7, 15, 7))
    return g


@pytest.mark.parametrize("spacing", [0.3, 0.2])  # 0.2: footprints past the shared box scatter directly
@pytest.mark.parametrize("kind", ["voxel", "corners", "box", "none"])
def test_sparse_part_of_a_gradient(kind, spacing):
    vol = inputs.head_neck_phantom(shape=(47, 44, 41), voxel_cm=0.3)
    rng = np.random.default_rng(8)
    bs = []
    for k, (g, c) in enumerate(inputs.four_pi_angles(5, seed=2)):
        b = inputs.single_beam(fmap=(7 + k, 9 - k), beamlet_cm=0.5, gantry_deg=float(g), couch_deg=float(c),
                               coll_deg=17.0 * k, iso=(0.2, -0.3, 0.1))
        b.fluence = rng.uniform(0.2, 1.0, b.fluence.shape).astype(np.float32)
        bs.append(b)
    gd = rng.standard_normal(vol.density.shape).astype(np.float32)
    gs = sparse(kind, vol.density.shape, rng)
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(inputs.make_physics(seed=1, spacing_cm=spacing), mode="exp")
        e.beam_dose(bs)
        both, dense, part = ([f.ravel().astype(np.float64) for f in e.beam_dose_adjoint(bs, g)] for g in (gd + gs, gd, gs))
    for a, d, p in zip(both, dense, part):
        np.testing.assert_allclose(p, a - d, rtol=0, atol=2e-5 * max(np.abs(d).max(), np.abs(a).max()))
        if kind == "none":
            assert not p.any()
