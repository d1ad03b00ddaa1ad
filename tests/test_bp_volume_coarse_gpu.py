"""Volumes of voxels several detector pixels wide (mr_backproject_volume_coarse) and volumes of
many blocks (two view shares a block) against the C oracle and the plain volume kernel.

Tolerance: on noise-like stacks a coordinate error of e pixels moves a sample by about 1.4 e of
its size; coordinates count from the block's first pixel, so they stay below 256 and carry about 3
FP32 roundings (256 * 2^-25 = 8e-6 each): rel-L2 <= 3.2e-5, and 5e-5 is the bar of the other
back-projection kernels. The two kernels round alike but for the cut of a block's footprint
(staged here, global memory there), so they are held to the same bar."""
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


def _case(orbit, store, A, rows, cols, dims, h, seed):
    rng = np.random.default_rng(seed)
    q = rng.normal(0.0, 1.0, (A, rows, cols)).astype(np.float32)
    origin = np.array([1.0, -2.0, 0.5]) - h * (np.asarray(dims) - 1) / 2.0
    grid = np.zeros(1, N.GRID_DTYPE)
    grid[0] = R.volume_grid_record(origin, h, dims)
    grid["scale"], grid["n_views"] = np.pi / A, A
    if orbit == "parallel":
        ang = np.arange(A) * np.pi / A
        ring = DeviceRing(q, R.parallel_view_maps(ang, 0.9, 1.1, rows, cols), N.MR_PARALLEL, store, None)
        stored = ring.stored.astype(np.float32)
        want = lambda pts: obp.bp_parallel(stored, np.cos(ang), np.sin(ang), 0.9, 1.1, pts, np.pi / A, 0.0)   # noqa: E731
    else:
        V = og.circular_cone_vectors(A, 600.0, 1000.0, 1.0, det_shift_u=0.6)
        if orbit == "tilted":
            V = V + rng.normal(0.0, 0.02, V.shape)
        K = of.cone_constants(V)
        ring = DeviceRing(q, R.cone_view_maps(R.cone_constants(V), rows, cols), N.MR_CONE, store, None)
        stored = ring.stored.astype(np.float32)
        want = lambda pts: obp.bp_cone(stored, K["s"], K["d"], K["uu"], K["vv"], K["n"], K["sdd"], K["sod"], pts,   # noqa: E731
                                       np.pi / A)
    return ring, grid, origin, want


def _run(ring, grid, dims, coarse, ranges=None):
    out = torch.full((int(np.prod(dims)),), float("nan"), dtype=torch.float32, device=ring.dev)
    status = torch.zeros(1, dtype=torch.int32, device=ring.dev)
    for i, (a, b) in enumerate(ranges or [(0, int(grid["n_views"][0]))]):
        g = grid.copy()
        g["view_begin"], g["n_views"], g["accumulate"] = a, b - a, int(i > 0)
        R.backproject_volume_device(ring.c, ring.views, g, out, torch.cuda.current_stream(), status=status,
                                    coarse=coarse)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return out.cpu().numpy().astype(np.float64)


# steps of 2 to 9 pixels: footprints inside a plain stage, between the two and past a coarse one
@pytest.mark.gpu
@pytest.mark.parametrize("dims,h", [((33, 17, 20), 1.2), ((32, 48, 16), 2.6), ((40, 20, 31), 3.6), ((24, 33, 16), 5.5)])
@pytest.mark.parametrize("orbit", ["aligned", "tilted", "parallel"])
@pytest.mark.parametrize("store", ["fp32", "bf16", "fp16"])
def test_coarse_volume(cuda, dims, h, orbit, store):
    ring, grid, origin, want = _case(orbit, store, 21, 160, 200, dims, h, 5)
    got = _run(ring, grid, dims, True)
    x, y, z = (origin[e] + h * np.arange(dims[e]) for e in range(3))
    X, Y, Z = np.meshgrid(x, y, z, indexing="ij")
    assert rel_l2(got, want(np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1))) < 5e-5
    assert rel_l2(got, _run(ring, grid, dims, False)) < 5e-5
    assert rel_l2(_run(ring, grid, dims, True, [(0, 1), (1, 9), (9, 21)]), got) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("orbit", ["aligned", "parallel"])
@pytest.mark.parametrize("coarse", [False, True])
def test_many_blocks(cuda, orbit, coarse):
    dims, h = (129, 127, 96), 1.0                                    # 9 x 8 x 6 blocks
    ring, grid, origin, want = _case(orbit, "fp32", 9, 100, 130, dims, h, 6)
    got = _run(ring, grid, dims, coarse).reshape(dims)
    at = np.random.default_rng(7).integers(0, dims, (20000, 3))
    assert rel_l2(got[tuple(at.T)], want(origin + h * at)) < 5e-5
    assert rel_l2(_run(ring, grid, dims, coarse, [(0, 1), (1, 9)]).reshape(dims), got) < 1e-6


def test_which_volumes_are_coarse():
    def rule(h, pixel, stretch=1.0):
        g = np.zeros(1, N.GRID_DTYPE)
        g[0] = R.volume_grid_record((0.0, 0.0, 0.0), h, (64, 64, 64))
        g["step_j"] *= stretch
        return R.is_coarse_volume(g[0], pixel)
    assert not rule(0.6, 0.2) and rule(0.8, 0.2) and rule(1.5, 0.2) and not rule(1.7, 0.2)
    assert rule(0.6, 0.2, 1.5) and not rule(0.6, float("nan"))
