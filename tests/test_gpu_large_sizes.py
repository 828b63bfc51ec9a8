"""Sizes at the end of what 32-bit indexes and a grid's second dimension hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel(kind, vt):
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    smax = Interface()
    smax.register_kernel("t", KernelType[kind], PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    return smax, smax.kernel("t")


def test_block_product_of_two_billion_blocks():
    """2^31 - 1 blocks of 1x1 in rows of 9, the last of them shorter."""
    import torch
    free, _ = torch.cuda.mem_get_info()
    if free < 70 << 30:
        pytest.skip("not enough device memory")
    nnz = (1 << 31) - 1
    n = (nnz + 8) // 9
    assert nnz % 9
    rp = torch.clamp(torch.arange(n + 1, dtype=torch.int64, device="cuda") * 9, max=nnz).int()
    col = torch.full((nnz,), 5, dtype=torch.int32, device="cuda")
    val = torch.ones(nnz, dtype=torch.float32, device="cuda")
    x = torch.full((n,), 2.0, dtype=torch.float32, device="cuda")
    y = torch.zeros_like(x)
    smax, k = _kernel("SPMV", np.float32)
    k.set_mat_bcrs(True)
    k.register_A(n, n, nnz, 1, 1, 1, 1, col, rp, val)
    k.register_B(n, x)
    k.register_C(n, y)
    k.initialize()
    k.apply()
    k.sync()
    smax.close()
    assert torch.equal(y, (rp[1:] - rp[:-1]).float() * 2)


def test_column_major_block_of_more_vectors_than_a_grid_is_high():
    """4.3 million vectors of 6 rows."""
    import torch
    n, kk = 6, 65535 * 64 + 70000
    rp = np.array([0, 2, 4, 5, 6, 8, 9], np.int32)
    col = np.array([0, 5, 1, 2, 2, 3, 4, 0, 5], np.int32)
    val = np.arange(1, 10, dtype=np.float32)
    A = torch.zeros(n, n, device="cuda")
    A[torch.from_numpy(np.repeat(np.arange(n), np.diff(rp))).cuda(), torch.from_numpy(col).long().cuda()] = torch.from_numpy(val).cuda()
    X = (torch.arange(n * kk, device="cuda") % 17).float()
    Y = torch.zeros_like(X)
    smax, k = _kernel("SPMM", np.float32)
    k.set_vec_row_major(False)
    k.register_A(n, n, len(col), col, rp, val)
    k.register_B(n, kk, X)
    k.register_C(n, kk, Y)
    k.initialize()
    k.apply()
    k.sync()
    smax.close()
    assert torch.equal(Y.view(kk, n), (X.view(kk, n).double() @ A.double().t()).float())
