"""The FFT filter's store loop writes a column group (one column per thread of a row pair)
without checks when the whole group lies inside the row. Row lengths just below, at and above a
multiple of the group (N/32 columns), with an even and an odd row count, against the NumPy
oracle; the bounds are those of an FP32 FFT against a float64 one: 1e-6 in the 2-norm, 3e-6 of
the peak for a single value."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import filter as of
from tomography_local_demo_b200 import recon as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 3])
@pytest.mark.parametrize("cols", [63, 65, 479, 480, 481, 512, 513, 1151, 1152, 1153, 2047, 2048])
def test_rows_at_the_edges_of_a_column_group(cuda, cols, rows):
    rng = np.random.default_rng(cols + rows)
    x = rng.normal(0, 1, (rows, 2, cols)).astype(np.float32)
    want = of.filter_rows(x, 0.5, "shepp-logan", exact64=True)
    got = R.filter_rows(x, 0.5, "shepp-logan")
    assert rel_l2(got, want) < 1e-6
    assert np.max(np.abs(np.asarray(got, np.float64) - want)) <= 3e-6 * np.abs(want).max()
