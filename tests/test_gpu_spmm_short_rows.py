"""SpMM of matrices with few entries a row: column-major blocks that run as one
product per column, blocks that do not, and small matrices on the grid kernel."""
import numpy as np
import pytest

from helpers import normwise, tol
from oracle.oracle import Oracle
from test_gpu_formats import gpu_spmm

pytestmark = pytest.mark.gpu
O = Oracle()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("n,long_row,k,row_major",
                         [((1 << 17) - 1, 9, 3, False), (1 << 17, 9, 3, False), (1 << 17, 9, 7, False),
                          (1 << 17, 9, 8, False), (3000, 2000, 8, False), (3000, 2000, 9, False),
                          (3000, 100, 32, True), (3000, 100, 5, True), ((1 << 17) + 1, 9, 32, True)])
def test_short_rows(vt, n, long_row, k, row_major):
    rng = np.random.default_rng(n + k)
    lens = rng.integers(0, 5, n)
    lens[n // 3] = long_row
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(vt)
    X = rng.uniform(-1, 1, n * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, row_major)
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=row_major)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("n,long_row", [((1 << 16) - 1, 40), (1 << 16, 40), ((1 << 18) - 1, 64), (1 << 18, 65), (3000, 700)])
@pytest.mark.parametrize("k", [2, 3, 8, 32])
def test_row_major_rules_choose_between_equals(vt, n, long_row, k):
    """Whichever kernel the sizes choose, the sums are the grid kernel's, bit for bit."""
    rng = np.random.default_rng(n + k)
    lens = rng.integers(0, 5, n)
    lens[[0, n // 3, n - 1]] = long_row
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(vt)
    X = rng.uniform(-1, 1, n * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, True)
    np.testing.assert_array_equal(Y, gpu_spmm(rp, col, val, X, k, True, variant=1))
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=True)) <= tol(vt)
