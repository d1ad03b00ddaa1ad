"""The Gaussian's line kernel (mr_gaussian_axis_f32) against an FP64 convolution where its runs of
16 outputs, pairs of lines and blocks of lines end, on both axes and on both sides of the length
from which lines are cut into blocks of 512 outputs.

Tolerance: an output is a chain of up to 2 K + 1 <= 1950 FP32 multiply-adds, about half of them
rounding at the result's size: sqrt(1000) * 2^-25 = 9.4e-7, so rel-L2 <= 1.5e-6."""
import numpy as np
import pytest
import torch

from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import preprocess as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 2])
@pytest.mark.parametrize("n,other,k", [(1, 3, 2), (5, 1, 1), (16, 17, 1), (17, 16, 1), (40, 5, 3), (255, 7, 3), (486, 33, 1),
                                       (1025, 3, 3), (1944, 9, 1)])
@pytest.mark.parametrize("sigma", [0.5, 1.0, 4.0])
def test_lines_against_fp64(cuda, axis, n, other, k, sigma):
    shape = (n, k, other) if axis == 0 else (other, k, n)
    x = np.random.default_rng(n + other).normal(1.0, 1.0, shape).astype(np.float32)
    pad = int(np.ceil(3 * sigma))
    g = P.gaussian_taps(n, pad, sigma)
    taps = torch.from_numpy(g.astype(np.float32)).cuda()
    t = torch.from_numpy(x).cuda()
    out = torch.full_like(t, float("nan"))
    N.check(N.load().mr_gaussian_axis_f32(P._void(t.data_ptr()), P._void(out.data_ptr()), *(shape[0], k, shape[2]), axis,
                                          pad, P._void(taps.data_ptr()), len(g),
                                          P._void(torch.cuda.current_stream().cuda_stream)), "gaussian")
    a = np.take(x.astype(np.float64), np.arange(-pad, n + pad).clip(0, n - 1), axis=axis)
    f = np.fft.rfftfreq(n + 2 * pad)
    w = np.exp(-2.0 * (np.pi * f * sigma) ** 2)
    y = np.fft.irfft(np.fft.rfft(a, axis=axis) * (w[:, None, None] if axis == 0 else w), n + 2 * pad, axis=axis)
    want = np.take(y, np.arange(pad, n + pad), axis=axis)
    assert np.linalg.norm(out.cpu().numpy() - want) <= 1.5e-6 * np.linalg.norm(want)
