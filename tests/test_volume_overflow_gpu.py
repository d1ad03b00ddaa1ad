"""The threshold's tails where one value is frequent at a bracket (its voxels are counted and not
kept), and volumes too large for the tails. Exact: thresholds bit-equal to the NumPy oracle, counts equal to NumPy's."""
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
    v = rng.normal(0.3, 0.2, n).astype(np.float32)
    if kind == "constant":
        v[:] = 0.7
    elif kind == "clipped":                              # half the voxels at the smallest value
        v = np.maximum(v, np.float32(0.3))
    elif kind == "ceiling":
        v = np.minimum(v, np.float32(0.3))
    elif kind == "bytes":
        v = np.round(np.clip(v, 0, 1) * 255).astype(np.float32)
    return v


@pytest.mark.parametrize("kind", ["constant", "clipped", "ceiling", "bytes", "noise"])
@pytest.mark.parametrize("n", [1000, 262147, 10000003])
def test_counts_and_threshold(cuda, kind, n):
    v = _volume(kind, n)
    t = torch.from_numpy(v).cuda()
    lib = N.load()
    ws = torch.empty(int(lib.mr_volume_workspace_bytes()), dtype=torch.uint8, device="cuda")
    st = (ctypes.c_uint64 * 4)()
    N.check(lib.mr_volume_tails(V(t.data_ptr()), n, 0.001, 0.9995, V(ws.data_ptr()), st, None), "tails")
    live = np.sort(v[v != 0])
    assert st[0] == len(live) and st[1] == 0
    # whole runs of equal voxels: a tail ends where the sorted values change
    for size, edge in ((st[2], live[st[2] - 1]), (st[3], live[len(live) - st[3]])):
        assert size in (np.count_nonzero(live <= edge), np.count_nonzero(live >= edge))
    ranks = sorted({0, int(0.001 * len(live)), len(live) // 2, int(0.9995 * len(live)), len(live) - 1})
    for k in ranks:
        r, out = (ctypes.c_int64 * 1)(k), torch.empty(1, device="cuda")
        rc = lib.mr_volume_tail_select_equal(r, 1, st, V(ws.data_ptr()), V(out.data_ptr()), None)
        if k < st[2] or k >= len(live) - st[3]:
            N.check(rc, "select")
            assert float(out) == live[k]
        else:
            assert rc == N.MR_ERR_UNSUPPORTED
    assert M.otsu_threshold(t) == om.otsu_threshold(v)


def test_volumes_past_the_tails(cuda, monkeypatch):
    v = _volume("noise", 300001)
    v[::7] = 0.0
    t = torch.from_numpy(v).cuda()
    want = M.otsu_threshold(t)
    monkeypatch.setattr(M, "TAIL_MAX_VOXELS", 300000)
    assert M.otsu_threshold(t) == want == om.otsu_threshold(v)
    with pytest.raises(IndexError):
        M.otsu_threshold(torch.zeros(400000, device="cuda"))
    v[5] = np.nan
    with pytest.raises(ValueError):
        M.otsu_threshold(torch.from_numpy(v).cuda())
