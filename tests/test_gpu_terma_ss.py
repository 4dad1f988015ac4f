"""Supersampled TERMA: a block walks a brick's 64 ss^3 sub-voxel centres 1024
at a time, so the factors around that size (a chunk per brick, voxels split
over two chunks, chunks per voxel) against the FP64 oracle.

Tolerance 1e-3 of Dmax, the engine's bound against the oracle: a mis-summed
centre is 1/ss^3 of a voxel's TERMA, far above it at the factors up to 5, and a
dropped chunk at 8 is a sixteenth.  The oracle in FP32 with the texture unit's
weights stays within 7e-4 of its FP64 form on these beams, so no centre sits
on a beamlet edge that rounding decides.
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def problem():
    vol = inputs.slab_phantom(22, 0.25)
    phys = inputs.make_physics(seed=6, spacing_cm=0.25)
    beam = inputs.single_beam(fmap=(3, 2), beamlet_cm=0.67, gantry_deg=24.0, couch_deg=11.0, coll_deg=7.0)
    beam.fluence = np.random.default_rng(12).uniform(0.2, 1.0, beam.fluence.shape).astype(np.float32)
    return vol, phys, beam


@pytest.mark.parametrize("ss", [2, 3, 4, 5, 8])
def test_supersampled_dose_vs_fp64_oracle(ss):
    vol, phys, beam = problem()
    with engine.Engine(0) as e:
        e.set_volume(vol)
        e.set_physics(phys, mode="exp")
        e.set_terma_supersampling(ss)
        dose = e.beam_dose([beam])
    ref, _ = Oracle(vol, phys, kernel_mode=2, ss_factor=ss).beam_dose(beam)
    assert np.abs(dose - ref).max() <= 1e-3 * ref.max()
