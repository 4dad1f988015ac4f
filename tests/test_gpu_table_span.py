"""The table mode's window sums over the field's part of each line against the
step-by-step walk: a single beamlet, a slit, a field that covers whole lines, a
field whose beamlets are mostly closed, and a long column whose lines pass the
kernel's last radii outside the field; lines of 16 lanes and of 32.

Tolerance: the two modes differ in the order of FP32 sums only, <= 1e-4 of the
maximum of dose and gradient (the bar between these two modes elsewhere).
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu

FIELDS = {"one": (1, 1, 0.5), "slit": (1, 12, 0.4), "cover": (50, 50, 0.5), "closed": (9, 8, 0.4), "column": (3, 2, 0.5)}


@pytest.mark.parametrize("name", sorted(FIELDS))
def test_span_sums_match_the_walk(name):
    fx, fy, cm = FIELDS[name]
    rng = np.random.default_rng(len(name))
    if name == "column":
        dens = np.ones((18, 700, 18), np.float32)
        dens[:, 200:320, :] = 0.25
        start = -0.5 * (np.array([18, 700, 18]) - 1) * 0.25 + np.array([0.013, 0.0, -0.011])
        vol = inputs.Volume(density=dens, voxel=np.full(3, 0.25), start=start, bbox_start=np.zeros(3, np.int64),
                            bbox_size=np.array([18, 700, 18], np.int64))
        angles = [(90.0, 0.0), (60.0, 10.0)]  # across the column: the kernel's reach ends along it
    else:
        vol = inputs.head_neck_phantom(shape=(61, 57, 52), voxel_cm=0.3)
        angles = [(0.0, 0.0), (37.0, -21.0)]
    bs = []
    for g, c in angles:
        b = inputs.single_beam(fmap=(fx, fy), beamlet_cm=cm, gantry_deg=g, couch_deg=c, coll_deg=13.0)
        b.fluence = rng.uniform(0.2, 1.0, b.fluence.shape).astype(np.float32)
        if name == "closed":
            b.fluence *= rng.random(b.fluence.shape) < 0.1
            b.fluence[0, -1] = 0.6
        bs.append(b)
    g = rng.standard_normal(vol.density.shape).astype(np.float32)
    out = []
    for mode in ("table", "walk"):
        with engine.Engine(0) as e:
            e.set_volume(vol)
            e.set_physics(inputs.make_physics(seed=1, spacing_cm=0.25), mode=mode)
            out.append((e.beam_dose(bs, per_beam=True), [f.ravel() for f in e.beam_dose_adjoint(bs, g)]))
    for k in range(len(bs)):
        for a, b in ((out[0][0][k], out[1][0][k]), (out[0][1][k], out[1][1][k])):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-4 * np.abs(b).max())
