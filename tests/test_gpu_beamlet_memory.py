"""The buffers of the directions that share a launch stay within the scratch
limit, the lists of sources and lines with the REV arrays: for a beamlet of 16 cm
the list of sources is as large as the arrays.

What does not depend on the limit (the packed grid, the column's rows and
values) is in the use at a limit of 1 MB, as is one direction, which is always
taken; device memory is counted in whole 2 MB pieces, one per buffer at most.
"""
import pytest

from endtoend_gb300 import engine, inputs

pytestmark = pytest.mark.gpu

MB = 1 << 20


def used(limit):
    import torch
    torch.zeros(1, device="cuda")
    with engine.Engine(0) as e:
        e.set_volume(inputs.slab_phantom(64, 0.25))
        e.set_physics(inputs.make_physics(seed=1, spacing_cm=0.25), mode="table")
        e.set_scratch_limit(limit)
        e.synchronize()
        before = torch.cuda.mem_get_info()[0]
        e.beamlet_columns_device(inputs.single_beam(fmap=(1, 1), beamlet_cm=16.0, gantry_deg=40.0))
        e.synchronize()
        return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("limit", [64 * MB, 128 * MB, 192 * MB])
def test_group_within_the_limit(limit):
    one = used(1 * MB)
    assert used(limit) <= limit + one
