"""Which entry each grid of a list goes to when point lists, wide grids and others come together
(host only: the library's launches are recorded, not run)."""
import types

import numpy as np
import pytest

from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import recon as R


class Pointer:
    cuda_stream = 0

    def __init__(self, at=4096):
        self.at = at

    def data_ptr(self):
        return self.at

    def record_stream(self, stream):
        pass


@pytest.mark.parametrize("slim", [False, True, None])
@pytest.mark.parametrize("kinds", ["www", "ww", "www.", "pww", "wpw.", "p.w.pw", "pp", "p.", "..", "pwpw", "s.", "ss", "pswp.s", "sw"])
def test_entries(monkeypatch, kinds, slim):
    """kinds: w = wide, p = points, s = slim where that is said grid by grid (slim None), . = another
    regular grid; grid k has k + 1 tiles."""
    box = np.array([40.0, 40.0, 40.0])
    grids = np.zeros(len(kinds), N.GRID_DTYPE)
    for k, kind in enumerate(kinds):
        grids[k] = R.plane_grid(box, (0, 0, 0), (0, 0, 1.0), 8)
        grids[k]["n_i"] = 32 * (k + 1)
        if kind == "p":
            grids[k]["flags"], grids[k]["n_i"], grids[k]["n_j"] = N.MR_GRID_POINTS, 1, 1024 * (k + 1)
    calls = []

    def entry(name):
        def launch(*args):
            calls.append((name, args[4]))
            return 0
        return launch
    lib = types.SimpleNamespace(**{n: entry(n) for n in ("mr_backproject", "mr_backproject_staged",
                                                         "mr_backproject_staged_slim", "mr_backproject_staged_wide")})
    native = types.SimpleNamespace(**{k: v for k, v in vars(N).items() if not k.startswith("__")})
    native.load = lambda: lib
    monkeypatch.setattr(R, "N", native)
    monkeypatch.setattr(R, "_struct_tensor", lambda *a: Pointer())
    R.backproject_device(None, Pointer(), grids, Pointer(), Pointer(), None,
                         wide=True if kinds == "www" else [k == "w" for k in kinds],
                         slim=[k == "s" for k in kinds] if slim is None else slim)
    forms = {"p": "mr_backproject", "w": "mr_backproject_staged_wide", "s": "mr_backproject_staged_slim",
             ".": "mr_backproject_staged"}
    if slim is not None:
        forms["s"] = forms["."] = forms["s" if slim else "."]
    want = dict.fromkeys(forms.values(), 0)
    for k, kind in enumerate(kinds):
        want[forms[kind]] += k + 1
    assert dict(calls) == {n: t for n, t in want.items() if t} and len(calls) == len(dict(calls))
