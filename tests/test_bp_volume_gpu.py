"""The volume kernel (mr_backproject_volume: blocks of 16^3 voxels, columns along j) against
the C oracle on noise-like stacks, at the block's edges, on orbits of both kinds (detector
rows along j or not), with footprints staged, too wide for a stage and off the detector.

Tolerance: on such stacks a coordinate error of e pixels moves a sample by about 1.4 e of its
size; coordinates of at most 64 pixels carry about 3 FP32 roundings (64 * 2^-24 = 4e-6 each),
so rel-L2 <= 5e-5, the bar of the other back-projection kernels, leaves a factor of two."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from gpu_helpers import DeviceRing
from oracle import bp as obp
from oracle import filter as of
from oracle import geometry as og
from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import recon as R


def _grid(dims, h, centre=(0.0, 0.0, 0.0)):
    origin = np.asarray(centre) - h * (np.asarray(dims) - 1) / 2.0
    g = np.zeros(1, N.GRID_DTYPE)
    g[0] = R.volume_grid_record(origin, h, dims)
    x, y, z = (origin[e] + h * np.arange(dims[e]) for e in range(3))
    X, Y, Z = np.meshgrid(x, y, z, indexing="ij")
    return g, np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1)


def _run(ring, grid, ranges, dims):
    out = torch.full((int(np.prod(dims)),), float("nan"), dtype=torch.float32, device=ring.dev)
    status = torch.zeros(1, dtype=torch.int32, device=ring.dev)
    for i, (a, b) in enumerate(ranges):
        grid["view_begin"], grid["n_views"], grid["accumulate"] = a, b - a, int(i > 0)
        R.backproject_volume_device(ring.c, ring.views, grid, out, torch.cuda.current_stream(), status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return out.cpu().numpy().astype(np.float64)


# dims around the block edge; h: footprints inside a stage, wider than one (4.5), block
# corners off the detector (dims 70 x 16 x 90)
@pytest.mark.gpu
@pytest.mark.parametrize("dims,h", [((16, 16, 16), 0.7), ((17, 31, 15), 0.9), ((33, 8, 49), 0.6), ((8, 64, 9), 0.5),
                                    ((70, 16, 90), 0.8), ((20, 24, 18), 4.5), ((40, 40, 40), 1.3)])
@pytest.mark.parametrize("orbit", ["aligned", "tilted", "parallel"])
@pytest.mark.parametrize("store", ["fp32", "bf16", "fp16"])
def test_volume_matches_oracle(cuda, dims, h, orbit, store):
    A, rows, cols = 37, 48, 64
    rng = np.random.default_rng(3)
    q = rng.normal(0.0, 1.0, (A, rows, cols)).astype(np.float32)
    grid, pts = _grid(dims, h, (1.0, -2.0, 0.5))
    grid["scale"] = np.pi / A
    shift = 0.0 if orbit == "aligned" else -1.3
    grid["cor_shift"] = shift
    if orbit == "parallel":
        ang = np.arange(A) * np.pi / A
        ring = DeviceRing(q, R.parallel_view_maps(ang, 0.9, 1.1, rows, cols), N.MR_PARALLEL, store,
                          np.full(A, 2.0) if store == "fp16" else None)
        want = obp.bp_parallel(ring.stored.astype(np.float32), np.cos(ang), np.sin(ang), 0.9, 1.1, pts, np.pi / A,
                               shift)
    else:
        V = og.circular_cone_vectors(A, 150.0, 250.0, 1.0, det_shift_u=0.6)
        if orbit == "tilted":
            V = V + rng.normal(0.0, 0.02, V.shape)
        K = of.cone_constants(V)
        ring = DeviceRing(q, R.cone_view_maps(R.cone_constants(V), rows, cols), N.MR_CONE, store,
                          np.full(A, 2.0) if store == "fp16" else None)
        want = obp.bp_cone(ring.stored.astype(np.float32), K["s"], K["d"] - shift * K["u"], K["uu"], K["vv"], K["n"],
                           K["sdd"], K["sod"], pts, np.pi / A)
    got = _run(ring, grid, [(0, A)], dims)
    assert rel_l2(got, want) < 5e-5
    # view ranges added up: the same sum to FP32 rounding (fewer views than CTAs of a cluster)
    assert rel_l2(_run(ring, grid, [(0, 3), (3, 20), (20, A)], dims), got) < 1e-6


def test_which_grids_go_to_the_volume_kernel():
    def rule(n_i, n_j, n_k, flags=0, count=1):
        g = np.zeros(count, N.GRID_DTYPE)
        g["n_i"], g["n_j"], g["n_k"], g["flags"] = n_i, n_j, n_k, flags
        return R.is_block_volume(g)
    assert rule(64, 64, 64) and rule(256, 203, 256)
    assert not rule(512, 512, 1)                             # a slice: 16 times the work
    assert not rule(24, 24, 24)                              # too few blocks to fill the GPU
    assert not rule(512, 512, 7) and rule(512, 512, 8)       # thin slabs keep the tiles
    assert not rule(64, 64, 64, N.MR_GRID_MASK_BOX) and not rule(1, 300000, 1, N.MR_GRID_POINTS)
    assert not rule(64, 64, 64, count=2) and not rule(0, 64, 64)
