"""The threshold's one-pass order statistics (mr_volume_tails / mr_volume_tail_select) and its
histogram, where their cases change: fewer voxels than the sample, nearly all zero, many equal
values (the kept tails overflow: the radix select over the volume takes over), ranges of few
representable values. Exact: thresholds bit-equal to the NumPy oracle, ranks equal to a sort."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import model as om
from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import model as M
from tomography_local_demo_b200.recon import ctypes_void as V

pytestmark = pytest.mark.gpu


def _volume(kind, n):
    rng = np.random.default_rng(n)
    if kind == "noise":
        return rng.normal(0.2, 0.3, n).astype(np.float32)
    if kind == "sparse":                                 # a few voxels other than zero
        v = np.zeros(n, np.float32)
        v[rng.integers(0, n, 1 + n // 5000)] = 1.0 + rng.random(1 + n // 5000).astype(np.float32)
        return v
    if kind == "levels":                                 # few distinct values, many of each
        return np.round(rng.normal(0, 1.2, n)).astype(np.float32)
    if kind == "two":
        return rng.choice(np.array([0.5, 1.0], np.float32), n)
    if kind == "close":                                  # a range of some thousand FP32 steps
        return (1000.0 + rng.integers(0, 3000, n) * 2.0 ** -13).astype(np.float32)
    return np.exp(rng.normal(0, 6, n)).astype(np.float32) * np.where(rng.random(n) < 0.4, -1, 1).astype(np.float32)


@pytest.mark.parametrize("kind", ["noise", "sparse", "levels", "two", "close", "wide"])
@pytest.mark.parametrize("n", [7, 65, 32767, 32769, 700001, 9000001])
def test_threshold_equals_oracle(cuda, kind, n):
    v = _volume(kind, n)
    # an odd start: the aligned body does not begin at the first voxel
    t = torch.from_numpy(np.concatenate([[0.0], v]).astype(np.float32)).cuda()[1:]
    for bins in (2, 512, 2048):
        assert M.otsu_threshold(t, bins) == om.otsu_threshold(v, bins)


@pytest.mark.parametrize("kind,n", [("noise", 3000001), ("levels", 100000), ("levels", 9000000), ("two", 9000000), ("wide", 40001)])
def test_tail_ranks_equal_sorted_values(cuda, kind, n):
    lib = N.load()
    v = _volume(kind, n)
    t = torch.from_numpy(v).cuda()
    ws = torch.empty(int(lib.mr_volume_workspace_bytes()), dtype=torch.uint8, device="cuda")
    st = (ctypes.c_uint64 * 4)()
    N.check(lib.mr_volume_tails(V(t.data_ptr()), n, 0.001, 0.9995, V(ws.data_ptr()), st, None), "tails")
    s = np.sort(v[v != 0])
    assert st[0] == len(s) and st[1] == 0
    ranks = [0, int(0.001 * len(s)), int(0.9995 * len(s)), len(s) - 1]
    r = (ctypes.c_int64 * 4)(*ranks)
    out = torch.empty(4, dtype=torch.float32, device="cuda")
    rc = lib.mr_volume_tail_select(r, 4, st, V(ws.data_ptr()), V(out.data_ptr()), None)
    if kind == "two":                                    # each tail is 4.5 M equal voxels: not kept
        assert rc == N.MR_ERR_UNSUPPORTED
    else:
        N.check(rc, "select")
        np.testing.assert_array_equal(out.cpu().numpy(), s[ranks])
    r[0] = len(s)
    assert lib.mr_volume_tail_select(r, 1, st, V(ws.data_ptr()), V(out.data_ptr()), None) == N.MR_ERR_INVALID
    r[0] = len(s) // 2                                   # between the tails
    if kind == "noise":
        assert lib.mr_volume_tail_select(r, 1, st, V(ws.data_ptr()), V(out.data_ptr()), None) == N.MR_ERR_UNSUPPORTED
