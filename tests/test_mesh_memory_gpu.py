"""marching_cubes where the card has no room for the workspace of the indexed mesh: the passes over
the cells give the same vertices and faces, bit for bit."""
import ctypes

import pytest
import torch

from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 40), (33, 34, 65), (70, 2, 31), (60, 61, 62)])
@pytest.mark.parametrize("iso", [0.4, 2.5, 9.0])
def test_cell_passes_equal_the_mesh(cuda, shape, iso):
    vol = torch.randn(shape, generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    want = M.marching_cubes(vol, iso, (-1.0, 2.0, 0.5), 0.3)
    got = M._cells_mesh(N.load(), vol, iso, (ctypes.c_double * 3)(-1.0, 2.0, 0.5), 0.3, torch.cuda.current_stream())
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


def test_no_room_for_the_workspace(cuda):
    x = torch.linspace(-1, 1, 400, device="cuda")
    vol = 0.3 - torch.sqrt(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2)
    want = [a.cpu() for a in M.marching_cubes(vol, 0.0)]
    need = N.load().mr_mesh_workspace_bytes(400, 400, 400)
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:                                                # what is in use now, and less than the workspace
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 0.9 * need) / total)
        held = []                                       # what the allocator still has in pieces that large
        with pytest.raises(torch.OutOfMemoryError):
            while len(held) < 10000:
                held.append(torch.empty(need, dtype=torch.uint8, device="cuda"))
        got = M.marching_cubes(vol, 0.0)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert len(want[1]) > 10000
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)
