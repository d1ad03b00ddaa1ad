"""The derivative kernels where a tile's footprint decides the path: wholly on the detector
(unchecked taps), across its border, off it; partial tiles; masked samples; enough tiles for
every cluster size. Against the float64 operator.

Tolerances: detector coordinates below 80 pixels carry about three FP32 roundings, 80 * 3 *
2^-24 = 1.5e-5 pixels, and smooth projections change by less than their own size a pixel, so
rel-L2 <= 5e-5 for values and view gradients; the slope of the bilinear interpolant jumps at
pixel borders, which 1.5e-5 of the samples cross, so 1e-3 for shift and tilt as in the other
derivative tests."""
import math

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


@pytest.mark.parametrize("n,zoom", [(32, 3.0), (33, 1.0), (31, 0.3), (200, 1.6), (97, 6.0)])
@pytest.mark.parametrize("pitch", [0, 5])
@pytest.mark.parametrize("tilt", [0.0, 0.006])
def test_footprints_against_float64(cuda, n, zoom, pitch, tilt):
    A, rows, cols = 10, 44, 75
    rng = np.random.default_rng(n)
    V = og.circular_cone_vectors(A, 150.0, 250.0, 1.0) + rng.normal(0, 0.01, (A, 12))
    maps = R.cone_view_maps(R.cone_constants(V), rows, cols)
    box = og.cone_volume_box(V, rows, cols) * 1.3            # wider than the detector sees
    grids = np.zeros(2, N.GRID_DTYPE)
    for k, (o, nrm) in enumerate([((2.0, -1.0, 0.5), (0.3, 0.5, 0.8)), ((0.0, 3.0, 0.0), (0.1, 1.0, 0.05))]):
        grids[k] = R.plane_grid(box, o, nrm, n, None, zoom, None, 0.0)
        grids[k]["out_offset"] = k * n * n
    views = torch.from_numpy(maps.view(np.uint8).copy()).cuda()
    op = BackprojectOp(views, N.MR_CONE, rows, cols, grids, 2 * n * n)
    q, y = smooth_field(A, rows, cols, 2 * n * n)
    qp = torch.full((A, rows, cols + pitch), float("nan"), device="cuda")      # the padding is never read
    qp[:, :, :cols] = q
    qp.requires_grad_(True)
    s = torch.tensor(0.7, dtype=torch.float64, requires_grad=True)
    t = torch.tensor(tilt, dtype=torch.float64, requires_grad=True)
    f = backproject(qp, s, t, op)
    gq, gs, gt = torch.autograd.grad((f.double() * y).sum(), (qp, s, t))
    q64 = q.double().requires_grad_(True)
    s64 = torch.tensor(0.7, dtype=torch.float64, device="cuda", requires_grad=True)
    t64 = torch.tensor(tilt, dtype=torch.float64, device="cuda", requires_grad=True)
    f64 = torch64_reference(q64, maps, op.grids_at(0.0, 0.0), s64, t64, rows, cols)
    wq, ws, wt = torch.autograd.grad((f64 * y).sum(), (q64, s64, t64))
    assert rel_l2(f.detach().cpu().numpy(), f64.detach().cpu().numpy()) < 5e-5
    assert rel_l2(gq[:, :, :cols].cpu().numpy(), wq.cpu().numpy()) < 5e-5
    assert pitch == 0 or float(gq[:, :, cols:].abs().max()) == 0.0
    assert abs(float(gs) - float(ws)) <= 1e-3 * abs(float(ws))
    assert abs(float(gt) - float(wt)) <= 1e-3 * abs(float(wt))
