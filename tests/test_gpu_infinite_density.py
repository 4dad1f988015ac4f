"""An opaque block given as infinite density: a ray that crosses it has an
infinite radiological path and no TERMA behind it, as with a density too large
to see through.  The rays also make crossings below the reference's length cut
inside the block (cudaSiddon.cu:20-115), which count nothing, not 0 x infinity.

So the dose is finite, and no more voxels have TERMA than behind a block of 1e30
g/cc, whose attenuation underflows to exactly 0 too.  (The doses themselves
differ: a filtered density is not a number where an infinite corner has weight
0, and the cones leave such a sample out.)
"""
import numpy as np
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ss", [1, 2])
@pytest.mark.parametrize("gantry,couch,iso", [(0.0, 0.0, (0.0, 0.0, 0.0)), (33.0, 17.0, (0.013, 0.007, -0.011)),
                                              (90.0, 0.0, (0.013, 0.007, -0.011))])
def test_opaque_block(ss, gantry, couch, iso):
    doses, counts = [], []
    for value in (np.inf, 1e30):
        vol = inputs.slab_phantom(32, 0.25)
        vol.density[:] = 1.0
        vol.density[14:17, 14:17, 14:17] = value
        beam = inputs.single_beam(fmap=(6, 6), beamlet_cm=0.5, gantry_deg=gantry, couch_deg=couch, iso=iso)
        with engine.Engine(0) as e:
            e.set_volume(vol)
            e.set_physics(inputs.make_physics(seed=3, spacing_cm=0.25), mode="exp")
            e.set_terma_supersampling(ss)
            doses.append(e.beam_dose([beam]))
            counts.append(e.beam_info(0)["terma_nonzero"])
    assert np.isfinite(doses[0]).all() and np.isfinite(doses[1]).all()
    assert 0 < counts[0] <= counts[1]
