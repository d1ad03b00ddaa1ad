"""The derivative kernels under each placement of a warp's samples: along j, along i (a grid whose j
is the rotation axis) and in patches (axial samples wider than 2.5 detector pixels); ragged sizes,
cone and parallel beams, one and many tiles. Against the float64 operator, with the tolerances of
the footprint tests (FP32 roundings of the detector coordinates)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import geometry as og
from test_autograd_gpu import smooth_field, torch64_reference
from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import recon as R
from tomography_local_demo_b200.autograd import BackprojectOp, backproject

pytestmark = pytest.mark.gpu


def transposed(g):
    """The same samples with i and j exchanged (the output transposed)."""
    h = g.copy()
    for a, b in (("step_i", "step_j"), ("mask_ei", "mask_ej")):
        h[a], h[b] = g[b], g[a]
    return h


@pytest.mark.parametrize("n", [1, 31, 33, 150])
@pytest.mark.parametrize("normal,turn,zoom", [((0.05, 1.0, 0.0), False, 1.3), ((0.05, 1.0, 0.0), True, 1.3),
                                              ((0.02, 0.0, 1.0), False, 0.0), ((0.3, 0.5, 0.8), True, 1.0)])
@pytest.mark.parametrize("kind", ["cone", "parallel"])
def test_lane_placements_against_float64(cuda, n, normal, turn, zoom, kind):
    A, rows, cols = 9, 44, 75
    rng = np.random.default_rng(n)
    if kind == "cone":
        V = og.circular_cone_vectors(A, 150.0, 250.0, 1.0) + rng.normal(0, 0.01, (A, 12))
        maps, code, box = R.cone_view_maps(R.cone_constants(V), rows, cols), N.MR_CONE, og.cone_volume_box(V, rows, cols)
    else:
        maps = R.parallel_view_maps(np.arange(A) * np.pi / A, 0.6, 0.6, rows, cols)
        code, box = N.MR_PARALLEL, np.array([0.3 * cols, 0.3 * cols, 0.3 * rows])
    # zoom 0: samples of 4 pixels (0.6 mm each at the axis)
    g = R.plane_grid(box, (0.4, -1.0, 0.5), normal, n, None if zoom else 2.4 * n, zoom or 1.0, None, 0.0)
    grids = np.array([transposed(g) if turn else g], dtype=N.GRID_DTYPE)
    op = BackprojectOp(torch.from_numpy(maps.view(np.uint8).copy()).cuda(), code, rows, cols, grids, n * n)
    q, y = smooth_field(A, rows, cols, n * n)
    q.requires_grad_(True)
    s = torch.tensor(0.7, dtype=torch.float64, requires_grad=True)
    t = torch.tensor(0.006, dtype=torch.float64, requires_grad=True)
    f = backproject(q, s, t, op)
    gq, gs, gt = torch.autograd.grad((f.double() * y).sum(), (q, s, t))
    q64 = q.detach().double().requires_grad_(True)
    s64, t64 = (torch.tensor(x, dtype=torch.float64, device="cuda", requires_grad=True) for x in (0.7, 0.006))
    f64 = torch64_reference(q64, maps, op.grids_at(0.0, 0.0), s64, t64, rows, cols)
    wq, ws, wt = torch.autograd.grad((f64 * y).sum(), (q64, s64, t64))
    assert float(wq.abs().max()) > 0
    assert rel_l2(f.detach().cpu().numpy(), f64.detach().cpu().numpy()) < 5e-5
    assert rel_l2(gq.cpu().numpy(), wq.cpu().numpy()) < 5e-5
    assert abs(float(gs) - float(ws)) <= 1e-3 * abs(float(ws)) + 1e-6 * float(y.abs().sum())
    assert abs(float(gt) - float(wt)) <= 1e-3 * abs(float(wt)) + 1e-4 * float(y.abs().sum())
