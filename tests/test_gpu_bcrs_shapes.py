"""BCRS SpMV over block shapes, short and long block rows, both in-block orders
and x at an address that is no multiple of 16 bytes: every kernel and every way
of reading x."""
import numpy as np
import pytest

from helpers import normwise, tol
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
O = Oracle()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("shape", [(3, 3, 3, 3), (2, 2, 2, 2), (4, 4, 4, 4), (5, 5, 5, 5), (2, 3, 3, 3), (6, 6, 6, 6),
                                   (7, 3, 7, 3), (3, 4, 4, 4), (8, 8, 8, 8), (1, 16, 1, 16), (16, 2, 16, 2),
                                   (11, 11, 11, 11), (12, 11, 12, 11)])
@pytest.mark.parametrize("col_major", [False, True])
@pytest.mark.parametrize("most", [4, 60])
@pytest.mark.parametrize("off", [0, 1])
def test_block_shapes_vs_oracle(vt, shape, col_major, most, off):
    import torch
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    bh, bw, hp, wp = shape
    nb = 300
    rng = np.random.default_rng(bh * 100 + bw + most)
    lens = rng.integers(0, most + 1, nb)
    lens[7] = 5 * most  # one long block row
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(nb, l, replace=False)) for l in lens]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col) * hp * wp).astype(vt)
    x = rng.uniform(-1, 1, nb * wp).astype(vt)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMV, PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    k = smax.kernel("k")
    k.set_mat_bcrs(True)
    k.set_block_column_major(col_major)
    k.register_A(nb, nb, len(col), bh, bw, hp, wp, col, rp, val)
    xd = torch.zeros(nb * wp + 8, dtype=torch.from_numpy(x).dtype, device="cuda")
    xd[off:off + nb * wp] = torch.from_numpy(x).cuda()
    yd = torch.zeros(nb * hp, dtype=xd.dtype, device="cuda")
    k.register_B(nb * wp + 8, xd)
    k.register_C(nb * hp, yd)
    k.initialize()
    for _ in range(2):
        k.apply(0, off, 0)
    k.sync()
    y_ref = O.spmv_bcrs(nb, bh, bw, hp, wp, rp, col, val, col_major, x)
    rows = np.concatenate([np.arange(r * hp, r * hp + bh) for r in range(nb)])
    assert normwise(yd.cpu().numpy()[rows], y_ref[rows]) <= tol(vt)
    smax.close()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("most", [2, 9])
def test_many_short_block_rows(vt, most):
    """Enough block rows for a thread each, shorter and longer than that path takes."""
    import torch
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    nb = 1024 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    rng = np.random.default_rng(most)
    lens = rng.integers(0, most + 1, nb)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, nb, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col) * 9).astype(vt)
    x, y = rng.uniform(-1, 1, nb * 3).astype(vt), np.zeros(nb * 3, vt)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMV, PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    k = smax.kernel("k")
    k.set_mat_bcrs(True)
    k.register_A(nb, nb, len(col), 3, 3, 3, 3, col, rp, val)
    k.register_B(nb * 3, x)
    k.register_C(nb * 3, y)
    k.run()
    smax.close()
    assert normwise(y, O.spmv_bcrs(nb, 3, 3, 3, 3, rp, col, val, False, x)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("nb,per_row,bs", [(9999, 1, 5), (10000, 1, 5), (10001, 1, 5), (40000, 4, 5), (51200, 5, 5),
                                           (43200, 3, 6), (13499, 1, 3), (13500, 1, 3), (9471, 12, 3), (9500, 32, 3),
                                           (9500, 33, 3), (33000, 1, 9)])
def test_thread_or_lanes_at_their_border(vt, nb, per_row, bs):
    """Block rows of one length, where the kernel changes with their number and size."""
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    rng = np.random.default_rng(nb)
    rp = (np.arange(nb + 1) * per_row).astype(np.int32)
    col = rng.integers(0, nb, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col) * bs * bs).astype(vt)
    x, y = rng.uniform(-1, 1, nb * bs).astype(vt), np.zeros(nb * bs, vt)
    smax = Interface()
    smax.register_kernel("k", KernelType.SPMV, PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    k = smax.kernel("k")
    k.set_mat_bcrs(True)
    k.register_A(nb, nb, len(col), bs, bs, bs, bs, col, rp, val)
    k.register_B(nb * bs, x)
    k.register_C(nb * bs, y)
    k.run()
    smax.close()
    assert normwise(y, O.spmv_bcrs(nb, bs, bs, bs, bs, rp, col, val, False, x)) <= tol(vt)
