"""CRS SpMV of matrices whose longest row decides the kernel: a few lanes per
row up to 32 entries (1, 2 or 4 lanes) if most rows are about as long, the
entry stream for the others and beyond."""
import numpy as np
import pytest

from helpers import normwise, tol
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
O = Oracle()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("longest", [1, 4, 5, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("n", [1, 255, 4097])
@pytest.mark.parametrize("shortest,empty", [(1.0, 0.0), (0.75, 0.1), (0.0, 0.0), (0.0, 0.6)])
def test_longest_row(vt, longest, n, shortest, empty):
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    rng = np.random.default_rng(longest * 10 + n)
    n_cols = 50
    lens = rng.integers(int(shortest * longest), longest + 1, n)
    lens[rng.random(n) < empty] = 0
    lens[n // 2] = longest
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n_cols, l, replace=False)) for l in lens]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(vt)
    x = rng.uniform(-1, 1, n_cols).astype(vt)
    y = np.full(n, 7, vt)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMV, PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    k = smax.kernel("k")
    k.register_A(n, n_cols, len(col), col, rp, val)
    k.register_B(n_cols, x)
    k.register_C(n, y)
    k.run()
    smax.close()
    assert normwise(y, O.spmv_crs(rp, col, val, x)) <= tol(vt)
    assert (y[lens == 0] == 0).all()


@pytest.mark.parametrize("longest", [7, 27])
def test_row_blocks_of_a_host_product(longest):
    """2^18 rows and more with host operands: the product runs in row blocks,
    each starting inside the matrix's arrays."""
    from smaxkernels_b200 import Interface, KernelType, PlatformType
    rng = np.random.default_rng(longest)
    n = (1 << 18) + 77
    lens = rng.integers(longest * 3 // 4, longest + 1, n)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col))
    x, y = rng.uniform(-1, 1, n), np.zeros(n)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMV, PlatformType.CUDA)
    k = smax.kernel("k")
    k.register_A(n, n, len(col), col, rp, val)
    k.register_B(n, x)
    k.register_C(n, y)
    for _ in range(2):
        k.run()
    smax.close()
    assert normwise(y, O.spmv_crs(rp, col, val, x)) <= 1e-12


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("longest", [8, 9, 32])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18])
@pytest.mark.parametrize("far", [False, True])
def test_columns_near_and_all_over(vt, longest, n, far):
    """Neighbouring rows' columns decide between the kernels from 2^18 rows on."""
    from helpers import gpu_spmv
    rng = np.random.default_rng(longest)
    lens = np.full(n, longest)
    lens[:5] = [0, 1, longest, 2, 0]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    rows = np.repeat(np.arange(n), lens)
    col = (rng.integers(0, n, rp[-1]) if far else np.minimum(rows + rng.integers(0, 99, rp[-1]), n - 1)).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(vt)
    x = rng.uniform(-1, 1, n).astype(vt)
    assert normwise(gpu_spmv(rp, col, val, x), O.spmv_crs(rp, col, val, x)) <= tol(vt)


@pytest.mark.parametrize("vt,n9", [(np.float64, 776722), (np.float64, 776724), (np.float32, 1165084)])
def test_narrow_rows_beyond_the_cache(vt, n9):
    """Rows of 9 on both sides of 80 MiB of entries, and as many of 27 a little wide."""
    from helpers import gpu_spmv
    rng = np.random.default_rng(n9)
    for longest, apart in ((9, 40), (27, 37)):
        n = n9 * 9 // longest
        rp = np.arange(n + 1, dtype=np.int32) * longest
        col = ((np.arange(n)[:, None] + apart * np.arange(longest)) % n).astype(np.int32).reshape(-1)
        val = rng.uniform(-1, 1, len(col)).astype(vt)
        x = rng.uniform(-1, 1, n).astype(vt)
        assert normwise(gpu_spmv(rp, col, val, x), O.spmv_crs(rp, col, val, x)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("longest,nnz", [(8, 1 << 20), (16, 1 << 20), (16, (1 << 20) - 16), (32, 1 << 20)])
@pytest.mark.parametrize("more", [0, 1])
def test_rows_that_share_banks(vt, longest, nnz, more):
    """2^20 entries and less, columns as wide apart as counts as narrow and one more,
    some rows shorter or empty."""
    from helpers import gpu_spmv
    n = nnz // longest + 110
    width = (80 if longest < 32 else 40) * longest + more
    rng = np.random.default_rng(longest)
    lens = np.full(n, longest)
    lens[100:200] = 0
    lens[300:320] = longest // 2
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    first = np.repeat(np.arange(n), lens)
    last = np.zeros(len(first), bool)
    last[rp[1:][lens > 0] - 1] = True
    step = np.where(last, width, rng.integers(0, width, len(first)))
    head = np.zeros(len(first), bool)
    head[rp[:-1][lens > 0]] = True
    col = (np.minimum(first, n - width - 1) + np.where(head, 0, step)).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(vt)
    x = rng.uniform(-1, 1, n).astype(vt)
    assert normwise(gpu_spmv(rp, col, val, x), O.spmv_crs(rp, col, val, x)) <= tol(vt)
