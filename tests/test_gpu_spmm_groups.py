"""SpMM with block widths that are no power of two, unaligned blocks, few rows,
and values beside the operands that must not be touched: the lane-group
kernel's lane counts, vector widths and panels, in both layouts."""
import numpy as np
import pytest

from helpers import normwise, rand_crs, tol
from oracle.oracle import Oracle
from test_gpu_formats import gpu_spmm

pytestmark = pytest.mark.gpu
O = Oracle()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [2, 5, 6, 7, 9, 10, 12, 20, 23, 24, 33, 48, 63, 65, 127, 130, 257, 530])
@pytest.mark.parametrize("row_major", [True, False])
def test_block_widths_vs_oracle(vt, k, row_major):
    rp, col, val = rand_crs(700, 20, k, vt=vt, empty_frac=0.1, long_rows=(600,))
    X = np.random.default_rng(k).uniform(-1, 1, 700 * k).astype(vt)
    Y = gpu_spmm(rp, col, val, X, k, row_major)
    assert normwise(Y, O.spmm(rp, col, val, X, k, row_major=row_major)) <= tol(vt)


@pytest.mark.parametrize("row_major,n,n_cols,maxlen",
                         [(True, 1, 9, 9), (True, 3, 500, 40), (True, 150, 40, 4), (True, 400, 300, 1),
                          (False, 1, 9, 9), (False, 3, 500, 40), (False, 300, 400, 5)])
def test_few_rows_and_rectangles(row_major, n, n_cols, maxlen):
    """Column-major blocks take A's row count as their leading dimension."""
    rp, col, val = rand_crs(n, maxlen, n, n_cols=n_cols)
    k = 6
    X = np.random.default_rng(n).uniform(-1, 1, n_cols * k)
    Y = gpu_spmm(rp, col, val, X, k, row_major, n_cols=n_cols)
    if row_major:
        ref = O.spmm(rp, col, val, X, k, row_major=True)
    else:
        ref = np.concatenate([O.spmm(rp, col, val, np.ascontiguousarray(X[v * n:v * n + n_cols]), 1) for v in range(k)])
    assert normwise(Y, ref) <= 1e-12


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k,off", [(4, 1), (8, 2), (12, 3), (5, 1)])
def test_offset_blocks_and_untouched_neighbours(vt, k, off):
    """X and Y shifted by `off` values (16-byte vectors do not apply), with
    NaN around the operands: nothing outside is read into a result or written."""
    import torch
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    n = 900
    rp, col, val = rand_crs(n, 12, k, vt=vt)
    X = np.random.default_rng(off).uniform(-1, 1, n * k).astype(vt)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMM, PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    kern = smax.kernel("k")
    kern.set_vec_row_major(True)
    xd = torch.full((n * k + 2 * k,), float("nan"), dtype=torch.from_numpy(X).dtype, device="cuda")
    yd = xd.clone()
    xd[off:off + n * k] = torch.from_numpy(X).cuda()
    kern.register_A(n, n, len(col), col, rp, val)
    kern.register_B(n + 2, k, xd)
    kern.register_C(n + 2, k, yd)
    kern.initialize()
    kern.apply(0, off, off)
    kern.sync()
    y = yd.cpu().numpy()
    assert normwise(y[off:off + n * k], O.spmm(rp, col, val, X, k)) <= tol(vt)
    assert np.isnan(y[:off]).all() and np.isnan(y[off + n * k:]).all()
    smax.close()


def test_infinity_in_an_unused_column():
    rp, col, val = rand_crs(200, 10, 3, n_cols=200)
    keep = col != 0
    rp = np.concatenate([[0], np.cumsum([keep[a:b].sum() for a, b in zip(rp[:-1], rp[1:])])]).astype(np.int32)
    col, val = col[keep], val[keep]
    for row_major in (True, False):
        X = np.ones((200, 3))
        X[0] = np.inf
        Xs = np.ascontiguousarray(X if row_major else X.T).reshape(-1)
        assert np.isfinite(gpu_spmm(rp, col.copy(), val.copy(), Xs, 3, row_major)).all()
