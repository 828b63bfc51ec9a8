"""Threads that each drive a kernel object of their own, on the same compiled
kernels with different amounts of shared memory."""
import threading

import numpy as np
import pytest

from helpers import normwise, rand_crs
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
O = Oracle()


def _together(jobs):
    """Runs the jobs in threads, starting together; raises what they raise."""
    gate, errors = threading.Barrier(len(jobs)), []

    def body(f):
        try:
            gate.wait()
            f()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    ts = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


def _interface(kind):
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    smax = Interface()
    smax.register_kernel("t", KernelType[kind], PlatformType.CUDA, IntType.INT32, FloatType.FLOAT64)
    return smax, smax.kernel("t")


def test_spmm_of_different_widths():
    import torch
    rp, col, val = rand_crs(2000, 14, 5, long_rows=(90,))
    jobs, checks = [], []
    for kk in (3, 8, 10):
        X = np.random.default_rng(kk).uniform(-1, 1, 2000 * kk)
        smax, k = _interface("SPMM")
        k.set_vec_row_major(True)
        xd = torch.from_numpy(X).cuda()
        yd = torch.zeros_like(xd)
        k.register_A(2000, 2000, len(col), col, rp, val)
        k.register_B(2000, kk, xd)
        k.register_C(2000, kk, yd)
        k.set_spmv_variant(2)
        k.initialize()

        def job(k=k):
            for _ in range(3000):
                k.apply()
            k.sync()
        jobs.append(job)
        checks.append((smax, yd, O.spmm(rp, col, val, X, kk, row_major=True)))
    _together(jobs)
    for smax, yd, ref in checks:
        assert normwise(yd.cpu().numpy(), ref) <= 1e-12
        smax.close()


def test_spgemm_of_different_row_lengths():
    jobs, checks = [], []
    for maxlen in (14, 60):
        A = rand_crs(600, maxlen, maxlen)
        smax, k = _interface("SPGEMM")
        rp, col, val = A
        k.register_A(600, 600, len(col), col, rp, val)
        k.register_B(600, 600, len(col), col, rp, val)
        k.register_C()
        k.initialize()

        def job(k=k):
            for _ in range(400):
                k.apply()
            k.finalize()
        jobs.append(job)
        checks.append((smax, k, O.spgemm(*A, *A, 600)))
    _together(jobs)
    for smax, k, (orp, ocol, oval) in checks:
        _, _, _, crp, ccol, cval = k.result()
        np.testing.assert_array_equal(crp, orp)
        np.testing.assert_array_equal(ccol, ocol)
        assert normwise(cval, oval) <= 1e-12
        smax.close()
