"""Tilt rotation (mr_rotate_f32): a thread samples up to eight views at once, a last group of
fewer views one by one. Blocks of 1 to 17 views must equal the views rotated one by one, bit for
bit, and the NumPy oracle. Tolerance against the oracle: the FP32 source coordinates (below 256)
carry at most four roundings of half an ulp, 2^-17 each, in either direction; values in [0, 1)
change by at most 1 a pixel, so 2 * 4 * 2^-17 = 6.1e-5."""
import numpy as np
import pytest
import torch

from oracle import filter as of
from tomography_local_demo_b200 import preprocess as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degrees", [0.3, -1.2, 40.0])
@pytest.mark.parametrize("rows,views,cols", [(33, 1, 127), (20, 7, 128), (65, 8, 129), (7, 9, 200), (5, 17, 31)])
def test_blocks_of_views(cuda, rows, views, cols, degrees):
    rng = np.random.default_rng(rows * views)
    x = rng.uniform(0, 1, (rows, views, cols)).astype(np.float32)
    got = P.rotate_projections(x, degrees)
    for a in range(views):
        np.testing.assert_array_equal(got[:, a:a + 1], P.rotate_projections(x[:, a:a + 1], degrees))
    assert np.max(np.abs(got - of.rotate_projections(x, degrees))) <= 6.1e-5


def test_a_view_of_nan_stays_alone(cuda):
    x = torch.ones((6, 9, 40), device=cuda)
    x[:, 3] = float("nan")
    got = P.rotate_projections(x, 0.3)
    rest = [a for a in range(9) if a != 3]
    assert torch.isfinite(got[:, rest]).all() and torch.isnan(got[2:4, 3, 1:39]).all()
