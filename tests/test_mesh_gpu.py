"""The indexed mesh of marching cubes (mr_mesh_plan / mr_mesh_emit) against the CPU oracle at
the sizes where its 32-point words, 256-word blocks and the rounds of its prefix sum begin and
end. Exact: the oracle rounds every FP32 operation alike and numbers vertices by grid edge."""
import numpy as np
import pytest
import torch

from oracle import model as om
from tomography_local_demo_b200 import model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 31), (2, 3, 32), (4, 3, 33), (3, 5, 64), (3, 4, 65), (17, 16, 97),
                                   (2, 129, 33), (1030, 1030, 2)])
@pytest.mark.parametrize("kind", ["noise", "nan", "all", "none"])
def test_mesh_equals_oracle(cuda, shape, kind):
    if kind != "noise" and np.prod(shape) > 100_000:
        pytest.skip("the large grid once")
    vol = np.random.default_rng(5).normal(size=shape).astype(np.float32)
    if kind == "nan":                                  # NaN counts as outside, infinities as values
        vol[np.random.default_rng(6).random(shape) < 0.1] = np.nan
        vol[np.random.default_rng(7).random(shape) < 0.05] = np.inf
    iso = {"all": -100.0, "none": 100.0}.get(kind, 0.25)
    P, F = M.marching_cubes(torch.from_numpy(vol).cuda(), iso, (1.0, -2.0, 0.5), 0.3)
    with np.errstate(all="ignore"):
        want_P, want_F = om.marching_cubes(vol, iso, (1.0, -2.0, 0.5), 0.3)
    assert P.dtype == torch.float32 and F.dtype == torch.int64
    np.testing.assert_array_equal(P.cpu().numpy(), want_P)
    np.testing.assert_array_equal(F.cpu().numpy(), want_F)
