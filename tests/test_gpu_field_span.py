"""The exp cone kernels walk only the part of a line that the beam's field can
reach, and the gathers visit only the cones whose lines it can reach: dose
against the FP64 oracle and the adjoint through the dot-product identity, for
fields that most lines miss, fields wider than the volume, oblique fields at a
corner, and voxels that are not cubes (where lines are not bounded).

Tolerances: dose 1e-3 of Dmax (the engine's bound against the FP64 oracle:
texture filter weights of 8 bits and FP32 geometry); <g, A f> = <A^T g, f> to
1e-4 of |g| |A f| (FP32 sums of up to 1e5 terms in both directions; a dropped
or doubled sample at a field edge is of order 1e-2).
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

CASES = [
    # shape xyz, voxel, spacing, map, beamlet, (gantry, couch, coll), iso, ss
    ((40, 37, 33), 0.25, 0.25, (1, 1), 0.31, (33.0, 17.0, 5.0), inputs.ISO_OFFSET_CM, 1),
    ((40, 37, 33), 0.25, 0.25, (1, 1), 0.31, (33.0, 17.0, 5.0), inputs.ISO_OFFSET_CM, 2),
    ((24, 31, 29), 0.3, 0.3, (9, 4), 2.5, (200.0, -25.0, 40.0), inputs.ISO_OFFSET_CM, 1),
    ((36, 30, 41), 0.25, 0.31, (3, 8), 0.33, (290.0, 30.0, 0.0), (3.013, -2.507, 3.991), 1),
    ((33, 35, 34), 0.3, 0.25, (2, 5), 0.4, (0.0, 0.0, 0.0), (-3.513, 0.207, -2.991), 1),
]


@pytest.mark.parametrize("shape,voxel,spacing,fmap,beamlet,angles,iso,ss", CASES)
@pytest.mark.parametrize("mode", ["exp", "table"])
def test_dose_and_adjoint_by_field(shape, voxel, spacing, fmap, beamlet, angles, iso, ss, mode):
    check(inputs.head_neck_phantom(shape=shape, voxel_cm=voxel), shape, spacing, fmap, beamlet, angles, iso, ss, mode)


@pytest.mark.parametrize("mode", ["exp", "table"])
def test_voxels_that_are_not_cubes(mode):
    shape = (37, 30, 33)
    vol = inputs.head_neck_phantom(shape=shape, voxel_cm=0.27)
    vol.voxel = np.array([0.31, 0.24, 0.27])
    vol.start = -0.5 * (np.array(shape) - 1) * vol.voxel
    check(vol, shape, 0.27, (4, 3), 0.4, (62.0, 21.0, 9.0), inputs.ISO_OFFSET_CM, 1, mode)


def check(vol, shape, spacing, fmap, beamlet, angles, iso, ss, mode):
    rng = np.random.default_rng(sum(shape))
    vol.density[:] = rng.uniform(0.9, 1.1, vol.density.shape)
    phys = inputs.make_physics(seed=3, spacing_cm=spacing)
    beam = inputs.single_beam(fmap=fmap, beamlet_cm=beamlet, gantry_deg=angles[0], couch_deg=angles[1],
                              coll_deg=angles[2], iso=iso)
    beam.fluence = rng.uniform(0.2, 1.0, beam.fluence.shape).astype(np.float32)
    g = rng.standard_normal(vol.density.shape).astype(np.float32)
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(phys, mode=mode)
        e.set_terma_supersampling(ss)
        dose = e.beam_dose([beam])
        fgrad = e.beam_dose_adjoint([beam], g)[0]
    ref, _ = Oracle(vol, phys, kernel_mode=2 if mode == "exp" else 0, ss_factor=ss).beam_dose(beam)
    assert ref.max() > 0
    assert np.abs(dose - ref).max() <= 1e-3 * ref.max()
    there = float((g.astype(np.float64) * dose).sum())
    back = float((fgrad.astype(np.float64) * beam.fluence).sum())
    assert abs(there - back) <= 1e-4 * np.linalg.norm(g.astype(np.float64)) * np.linalg.norm(dose.astype(np.float64))
