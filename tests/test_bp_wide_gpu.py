"""mr_backproject_staged_wide: the same images as mr_backproject_staged bit for bit, whatever the
footprints of the tiles (inside a stage, in a wide box, larger than any, across the detector's
border, off it), and the rule that sends grids there. The staged kernel itself is held against
the oracle in the other back-projection tests."""
import numpy as np
import pytest
import torch

from gpu_helpers import DeviceRing
from oracle import geometry as og
from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import recon as R


@pytest.mark.gpu
@pytest.mark.parametrize("store", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("kind", ["cone", "parallel"])
def test_wide_boxes_change_nothing(cuda, store, kind):
    A, rows, cols = 29, 90, 420
    rng = np.random.default_rng(9)
    q = rng.normal(0, 1, (A, rows, cols)).astype(np.float32)
    if kind == "cone":
        V = og.circular_cone_vectors(A, 440.0, 680.0, 0.3) + rng.normal(0, 0.01, (A, 12))
        maps = R.cone_view_maps(R.cone_constants(V), rows, cols)
        code, pixel = N.MR_CONE, 0.3 * 440.0 / 680.0
    else:
        maps = R.parallel_view_maps(np.arange(A) * np.pi / A, 0.2, 0.2, rows, cols)
        code, pixel = N.MR_PARALLEL, 0.2
    ring = DeviceRing(q, maps, code, store, np.full(A, 2.0) if store == "fp16" else None)
    box = np.array([40.0, 40.0, 9.0])
    grids = []
    # detector pixels a sample: 1.5 (staged) to 14 (global memory), axial and oblique
    for pitch in (1.5, 2.4, 3.0, 4.2, 5.5, 7.0, 14.0):
        for nrm in ((0.0, 0.0, 1.0), (0.1, -0.05, 1.0), (0.2, 1.0, 0.1)):
            n = 45
            grids.append(R.plane_grid(box, (1.0, 2.0, 0.4), nrm, n, n * pitch * pixel))
    grids = np.array(grids, dtype=N.GRID_DTYPE)
    grids["out_offset"] = np.cumsum([0] + [45 * 45] * (len(grids) - 1))
    grids["n_views"], grids["scale"], grids["cor_shift"] = A, np.pi / A, 0.7
    images = []
    # no grid, every grid, and two of three (two launches) through the wide variant
    for wide in (None, [True] * len(grids), [k % 3 > 0 for k in range(len(grids))]):
        out = torch.full((len(grids) * 45 * 45,), float("nan"), dtype=torch.float32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        R.backproject_device(ring.c, ring.views, grids, out, torch.cuda.current_stream(), out.device, status=status,
                             band_axis=(0.0, 0.0, 1.0), wide=wide)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        images.append(out.cpu().numpy())
    assert np.abs(images[0]).max() > 0 and np.isfinite(images[0]).all()
    np.testing.assert_array_equal(images[0], images[1])
    np.testing.assert_array_equal(images[0], images[2])


def test_which_grids_are_wide():
    g = np.zeros(4, N.GRID_DTYPE)
    g["step_i"] = [(0, 1.0, 0), (0, 0.5, 0), (0, 0, 5.0), (0.6, 0.6, 3.0)]
    g["step_j"] = [(0.2, 0, 0), (0.2, 0, 0), (0.2, 0, 0), (0.2, 0, 0)]
    assert [R.is_wide(x, (0.0, 0.0, 1.0), 0.8) for x in g] == [True, False, False, True]
    assert [R.is_wide(x, (0.0, 1.0, 0.0), 0.8) for x in g] == [False, False, True, True]
    assert not any(R.is_wide(x, None, 0.8) for x in g)
