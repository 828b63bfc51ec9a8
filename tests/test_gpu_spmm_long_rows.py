"""Column-major SpMM of rows far longer than the others, which are cut into
pieces: lengths at the edges of a piece and of its larger size, every layout of
lanes, values that are not finite, and sums no further from 64 bits than those
of the products per column that the block replaces."""
import numpy as np
import pytest

from helpers import gpu_spmv, normwise, tol
from oracle.oracle import Oracle
from test_gpu_formats import gpu_spmm

pytestmark = pytest.mark.gpu
O = Oracle()


def _matrix(lens, seed, vt):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, len(lens), rp[-1]).astype(np.int32)
    return rp, col, rng.uniform(-1, 1, rp[-1]).astype(vt)


EDGES = [127, 128, 129, 255, 256, 257, 511, 513, 1023, 1025, 4096]


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 8, 9, 17, 31, 33, 64, 65, 130, 300])
def test_piece_edges_vs_oracle(vt, k):
    lens = np.full(3000, 5)
    lens[np.arange(len(EDGES)) * 251 + 7] = EDGES
    rp, col, val = _matrix(lens, k, vt)
    X = np.random.default_rng(k).uniform(-1, 1, 3000 * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, False)
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=False)) <= tol(vt)


@pytest.mark.parametrize("length", [128 * 1024, 128 * 1024 + 1, 600001])
def test_one_very_long_row(length):
    lens = np.full(9000, 6)
    lens[4000] = length
    rp, col, val = _matrix(lens, 1, np.float64)
    X = np.random.default_rng(2).uniform(-1, 1, 9000 * 6)
    Y = gpu_spmm(rp, col, val, X, 6, False)
    assert normwise(Y, O.spmm(rp, col, val, X, 6, row_major=False)) <= tol(np.float64)


def test_first_last_and_only_rows():
    for lens in ([700, 0, 2, 0, 700], [3000], [0] * 40 + [500], [500] + [0] * 40):
        rp, col, val = _matrix(np.array(lens), 3, np.float64)
        n = len(lens)
        X = np.random.default_rng(4).uniform(-1, 1, n * 5)
        Y = gpu_spmm(rp, col, val, X, 5, False)
        assert normwise(Y, O.spmm(rp, col, val, X, 5, row_major=False)) <= tol(np.float64), lens


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite(vt, bad):
    lens = np.full(2000, 9)
    lens[[5, 900]] = [1500, 60]
    rp, col, val = _matrix(lens, 5, vt)
    col[rp[5]], col[rp[900]], col[rp[1500]] = 77, 78, 79
    val[[rp[5], rp[900], rp[1500]]] = 1
    X = np.random.default_rng(6).uniform(-1, 1, (4, 2000)).astype(vt)
    X[1, [77, 78, 79]] = bad
    Y = gpu_spmm(rp, col, val, X.reshape(-1), 4, False)
    np.testing.assert_array_equal(np.isnan(Y), np.isnan(O.spmm(rp, col, val, X.reshape(-1), 4, row_major=False)))
    got = Y.reshape(4, 2000)[1, [5, 900, 1500]]
    assert np.isnan(got).all() if np.isnan(bad) else (got[~np.isnan(got)] == bad).all()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("lens", ["mixed", "27", "400", "2000"])
@pytest.mark.parametrize("k", [8, 40, 200])
def test_sums_no_worse_than_the_products_per_column(vt, lens, k):
    rng = np.random.default_rng(7)
    n = 6000 if k == 8 else 1500
    lens = {"mixed": np.exp(rng.normal(2.3, 1.2, n)).astype(int) + 1, "27": np.full(n, 27), "400": np.full(n, 400),
            "2000": np.where(np.arange(n) % 10 == 0, 2000, 1200)}[lens]
    rp, col, val = _matrix(lens, 8, vt)
    X = rng.uniform(-1, 1, (k, n)).astype(vt)
    Y = gpu_spmm(rp, col, val, X.reshape(-1), k, False).reshape(k, n)
    P = np.stack([gpu_spmv(rp, col, val, X[v]) for v in range(k)])
    xl = X.astype(np.longdouble)
    ref = np.stack([np.add.reduceat(val.astype(np.longdouble) * xl[v][col], rp[:-1]) for v in range(k)])
    block, products = (np.sqrt(np.mean((A - ref).astype(np.float64) ** 2)) for A in (Y, P))
    assert block <= products, (block, products)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [2, 3, 4])
@pytest.mark.parametrize("n,most", [(32767, 90), (32768, 90), (32768, 600), (50000, 8)])
def test_few_vectors_where_the_products_begin(vt, k, n, most):
    """2^18 entries, less and more, rows uneven, far longer or all equal."""
    lens = np.full(n, 8)
    lens[0] = most
    lens[1:1 + most] -= most > 8
    rp, col, val = _matrix(lens, k, vt)
    X = np.random.default_rng(9).uniform(-1, 1, n * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, False)
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=False)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("n,length", [(65535, 8), (65536, 8), (32767, 64), (32768, 63), (32768, 64),
                                       (5000, 64), (600, 512)])
def test_even_rows_where_the_products_begin(vt, k, n, length):
    """2^19 and 2^21 entries, less and more, in rows on both sides of 64; a few
    longer ones by a quarter, or just more."""
    lens = np.full(n, length)
    lens[:20] += length // 4 + (k == 3)
    lens[20:40] -= length // 4 + (k == 3)
    rp, col, val = _matrix(lens, k, vt)
    X = np.random.default_rng(10).uniform(-1, 1, n * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, False)
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=False)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("n,k", [((1 << 21) - 1, 3), (1 << 21, 3), ((1 << 22) - 1, 5), (1 << 22, 5), (1 << 22, 7)])
def test_many_short_rows_where_the_products_begin(vt, n, k):
    """2^21 and 2^22 rows of four entries, and one less."""
    rng = np.random.default_rng(k)
    rp = np.arange(0, 4 * n + 1, 4, dtype=np.int32)
    col = rng.integers(0, n, 4 * n).astype(np.int32)
    val = rng.uniform(-1, 1, 4 * n).astype(vt)
    X = rng.uniform(-1, 1, n * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, False).reshape(k, n)
    for v in range(k):
        ref = (val.astype(np.float64) * X[v * n:(v + 1) * n][col]).reshape(n, 4).sum(1)
        assert normwise(Y[v], ref) <= tol(vt)
