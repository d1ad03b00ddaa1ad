"""The Gaussian's line kernel against an FP64 convolution on long axes, on both sides of the lengths
at which a block takes 8 lines instead of 16 and 4 instead of 8.

Tolerance: a chain of up to 2 K + 1 = 7001 FP32 multiply-adds, about half of them rounding at the
result's size: sqrt(3500) * 2^-25 = 1.8e-6, so rel-L2 <= 2.7e-6."""
import numpy as np
import pytest
import torch

from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import preprocess as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 2])
@pytest.mark.parametrize("n,other,k", [(1270, 3, 1), (1290, 5, 1), (3480, 3, 1), (3520, 5, 1), (4096, 9, 1), (4881, 2, 3),
                                       (6000, 3, 1), (6990, 5, 1)])
def test_long_lines_against_fp64(cuda, axis, n, other, k):
    sigma, pad = 1.0, 3
    shape = (n, k, other) if axis == 0 else (other, k, n)
    x = np.random.default_rng(n).normal(1.0, 1.0, shape).astype(np.float32)
    g = P.gaussian_taps(n, pad, sigma)
    assert len(g) > 0.49 * n
    taps, t = torch.from_numpy(g.astype(np.float32)).cuda(), torch.from_numpy(x).cuda()
    out = torch.full_like(t, float("nan"))
    N.check(N.load().mr_gaussian_axis_f32(P._void(t.data_ptr()), P._void(out.data_ptr()), *shape, axis, pad,
                                          P._void(taps.data_ptr()), len(g),
                                          P._void(torch.cuda.current_stream().cuda_stream)), "gaussian")
    a = np.take(x.astype(np.float64), np.arange(-pad, n + pad).clip(0, n - 1), axis=axis)
    f = np.fft.rfftfreq(n + 2 * pad)
    w = np.exp(-2.0 * (np.pi * f * sigma) ** 2)
    y = np.fft.irfft(np.fft.rfft(a, axis=axis) * (w[:, None, None] if axis == 0 else w), n + 2 * pad, axis=axis)
    want = np.take(y, np.arange(pad, n + pad), axis=axis)
    assert np.linalg.norm(out.cpu().numpy() - want) <= 2.7e-6 * np.linalg.norm(want)
