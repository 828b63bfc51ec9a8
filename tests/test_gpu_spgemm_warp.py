"""SpGEMM rows on the warp hash path (tables of 512 to 8192 slots) around the
product counts where the path changes, and the download of large products."""
import numpy as np
import pytest

from helpers import normwise, tol
from oracle.oracle import Oracle
from test_gpu_spgemm import gpu_spgemm

pytestmark = pytest.mark.gpu
O = Oracle()


def _b_matrix(rng, vt, n_cols, long_len, sort):
    """400 rows: 200 of long_len entries, then 200 of one."""
    rows = [rng.choice(n_cols, long_len if i < 200 else 1, replace=False) for i in range(400)]
    if sort:
        rows = [np.sort(r) for r in rows]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    return rp, col, rng.uniform(-1, 1, len(col)).astype(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("long_len,sort", [(31, True), (32, False), (37, True)])
@pytest.mark.parametrize("n_cols", [40, 3000])
def test_spgemm_rows_at_the_bin_edges(vt, long_len, sort, n_cols):
    """Rows of A with exactly P products, P at, below and above each table's
    limit, mixing long and one-entry rows of B (so steps of 32 products span
    several B rows and repeat columns within a step when n_cols is small);
    pattern bit-exact, values in the product order of the oracle."""
    rng = np.random.default_rng(long_len + n_cols)
    B = _b_matrix(rng, vt, n_cols, long_len, sort)
    rows = []
    for P in (0, 1, 64, 65, 96, 255, 256, 257, 767, 768, 769, 1536, 1537, 3072, 3073, 6144, 6145):
        for _ in range(3):
            q, r = divmod(P, long_len)
            if q > 200:  # more products than the distinct long rows give
                q, r = 200, min(200, P - 200 * long_len)
            rows.append(rng.permutation(np.concatenate([rng.choice(200, q, replace=False),
                                                        200 + rng.choice(200, r, replace=False)])))
    arp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    acol = np.concatenate(rows).astype(np.int32)
    A = (arp, acol, rng.uniform(-1, 1, len(acol)).astype(vt))
    n_rows, nc, nnz, rp, col, val = gpu_spgemm(A, B, 400, n_cols)
    orp, ocol, oval = O.spgemm(*A, *B, n_cols)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(col, ocol)
    assert normwise(val, oval) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("nnz", [(4 << 20) // 12 - 4096, 1_000_003])
def test_large_product_is_downloaded_whole(vt, nnz):
    """I * B = B, with C's arrays below and above the size from which the
    download is cut into pieces, and no multiple of a piece; the arrays stay
    valid after the kernel object is gone and can be written."""
    rng = np.random.default_rng(nnz)
    n = 5000
    lens = np.full(n, nnz // n)
    lens[: nnz - lens.sum()] += 1
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = (np.arange(nnz) - np.repeat(rp[:-1].astype(np.int64), lens)).astype(np.int32)
    val = rng.uniform(-1, 1, nnz).astype(vt)
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, vt))
    _, _, got, crp, ccol, cval = gpu_spgemm(eye, (rp, col, val), n, n)
    assert got == nnz
    np.testing.assert_array_equal(crp, rp)
    np.testing.assert_array_equal(ccol, col)
    np.testing.assert_array_equal(cval, val)
    cval[-1] = 2
    assert cval[-1] == 2


@pytest.mark.parametrize("vt", [np.float64, np.float32])
def test_rows_of_every_size_at_once(vt):
    """Rows for every table of the warps and for tables in global memory, which run
    beside each other; repeated, and with the sizes in another order."""
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    rng = np.random.default_rng(15)
    n = 1200
    lens = rng.choice([1, 8, 20, 40, 70, 120, 260], n)
    for order in (np.argsort(lens), rng.permutation(n)):
        ls = lens[order]
        rp = np.concatenate([[0], np.cumsum(ls)]).astype(np.int32)
        col = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in ls]).astype(np.int32)
        val = rng.uniform(-1, 1, len(col)).astype(vt)
        orp, ocol, oval = O.spgemm(rp, col, val, rp, col, val, n)
        smax = Interface()
        smax.register_kernel("k", KernelType.SPGEMM, PlatformType.CUDA, IntType.INT32,
                             FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
        k = smax.kernel("k")
        k.register_A(n, n, len(col), col, rp, val)
        k.register_B(n, n, len(col), col, rp, val)
        k.register_C()
        for _ in range(3):
            k.run()
            _, _, _, crp, ccol, cval = k.result()
            np.testing.assert_array_equal(crp, orp)
            np.testing.assert_array_equal(ccol, ocol)
            assert normwise(cval, oval) <= tol(vt)
        smax.close()
