"""mr_backproject_staged_slim against mr_backproject_staged, each asked for by name: the same images
bit for bit, over ragged sizes, masks, footprints of every kind, few and many tiles and view ranges
added up. The staged kernel itself is held against the oracle in the other back-projection tests."""
import numpy as np
import pytest
import torch

from gpu_helpers import DeviceRing
from oracle import geometry as og
from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import recon as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("store", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("kind", ["cone", "parallel"])
@pytest.mark.parametrize("count", [1, 40])
def test_slim_changes_nothing(cuda, store, kind, count):
    A, rows, cols = 23, 64, 140
    rng = np.random.default_rng(count)
    q = rng.normal(0, 1, (A, rows, cols)).astype(np.float32)
    if kind == "cone":
        V = og.circular_cone_vectors(A, 150.0, 250.0, 1.0) + rng.normal(0, 0.01, (A, 12))
        maps, code = R.cone_view_maps(R.cone_constants(V), rows, cols), N.MR_CONE
    else:
        maps, code = R.parallel_view_maps(np.arange(A) * np.pi / A, 0.6, 0.6, rows, cols), N.MR_PARALLEL
    ring = DeviceRing(q, maps, code, store, np.full(A, 2.0) if store == "fp16" else None)
    box = np.array([45.0, 40.0, 24.0])
    grids, off = [], 0
    for _ in range(count):
        n = int(rng.integers(31, 128))
        nrm = rng.normal(size=3)
        g = R.plane_grid(box, rng.uniform(-8, 8, 3), nrm / np.linalg.norm(nrm), n, None, float(rng.uniform(0.3, 6.0)))
        g["out_offset"], g["cor_shift"] = off, rng.uniform(-2, 2)
        grids.append(g)
        off += n * n
    grids = np.array(grids, dtype=N.GRID_DTYPE)
    grids["scale"] = np.pi / A
    images = []
    for slim in (False, True):
        out = torch.full((off,), float("nan"), dtype=torch.float32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        for a, b in ((0, 2), (2, 15), (15, A)):        # fewer views than a cluster's CTAs first
            grids["view_begin"], grids["n_views"], grids["accumulate"] = a, b - a, int(a > 0)
            R.backproject_device(ring.c, ring.views, grids, out, torch.cuda.current_stream(), out.device, status=status,
                                 slim=slim)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        images.append(out.cpu().numpy())
    assert np.abs(images[0]).max() > 0 and np.isfinite(images[0]).all()
    np.testing.assert_array_equal(*images)
