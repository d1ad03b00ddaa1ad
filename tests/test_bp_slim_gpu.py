"""The staged back-projection with four consumer warps a tile (launches of many tiles) against
the same grids launched one by one (few tiles: eight warps): the same images bit for bit, over
ragged sizes, masks, footprints of every kind and view ranges added up. The one-by-one launches
are held against the oracle in the other back-projection tests."""
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
def test_many_tiles_equal_few(cuda, store, kind):
    A, rows, cols = 31, 70, 150
    rng = np.random.default_rng(12)
    q = rng.normal(0, 1, (A, rows, cols)).astype(np.float32)
    if kind == "cone":
        V = og.circular_cone_vectors(A, 150.0, 250.0, 1.0) + rng.normal(0, 0.01, (A, 12))
        maps, code = R.cone_view_maps(R.cone_constants(V), rows, cols), N.MR_CONE
    else:
        maps, code = R.parallel_view_maps(np.arange(A) * np.pi / A, 0.6, 0.6, rows, cols), N.MR_PARALLEL
    ring = DeviceRing(q, maps, code, store, np.full(A, 2.0) if store == "fp16" else None)
    box = np.array([45.0, 40.0, 24.0])
    grids, off = [], 0
    for k in range(60):                                # 60 grids of 4 to 16 tiles: 500 to 600 in all
        n = int(rng.integers(33, 128))
        nrm = rng.normal(size=3)
        g = R.plane_grid(box, rng.uniform(-8, 8, 3), nrm / np.linalg.norm(nrm), n, None, float(rng.uniform(0.4, 6.0)))
        g["out_offset"], g["cor_shift"] = off, rng.uniform(-2, 2)
        grids.append(g)
        off += n * n
    grids = np.array(grids, dtype=N.GRID_DTYPE)
    grids["scale"] = np.pi / A
    assert len(N.plan_tiles(grids)) > 400

    def run(parts):
        out = torch.full((off,), float("nan"), dtype=torch.float32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        for a, b in ((0, 2), (2, 20), (20, A)):        # fewer views than a cluster's CTAs first
            for p in parts:
                p = p.copy()
                p["view_begin"], p["n_views"], p["accumulate"] = a, b - a, int(a > 0)
                R.backproject_device(ring.c, ring.views, p, out, torch.cuda.current_stream(), out.device, status=status)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        return out.cpu().numpy()

    many = run([grids])
    few = run([grids[k:k + 1] for k in range(len(grids))])
    assert np.abs(many).max() > 0 and np.isfinite(many).all()
    np.testing.assert_array_equal(many, few)
