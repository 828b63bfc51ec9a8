"""Level sweeps of triangular solves (SpTRSV, SpTRSM, batches) at the sizes
where their layout changes: rows of one to many entries, levels at the CTA
sizes' edges and wider than a CTA, rows too wide for the shared-memory stage,
sources older than the ring of recent solutions, and new values on the same
pattern.  Checked against the oracle; blocks of right-hand sides bit for bit
against the level launches, whose arithmetic they share."""
import numpy as np
import pytest

from helpers import normwise, tol
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
O = Oracle()


def level_matrix(sizes, width, seed, vt, reach=None):
    """Lower triangle whose dependency levels have the given sizes: a row has
    an entry in the level before its own and up to width - 1 others among the
    `reach` rows before its level; the diagonal is last."""
    rng = np.random.default_rng(seed)
    starts = np.concatenate([[0], np.cumsum(sizes)])
    rp, cols = [0], []
    for s, m in enumerate(sizes):
        a = int(starts[s])
        lo = 0 if reach is None else max(0, a - reach)
        for r in range(a, a + m):
            c = []
            if s:
                k = int(rng.integers(1, width + 1))
                c = {int(rng.integers(starts[s - 1], a))}
                c |= set(int(v) for v in rng.integers(lo, a, k - 1))
                c = sorted(c)
            cols += c + [r]
            rp.append(len(cols))
    rp, col = np.array(rp, np.int32), np.array(cols, np.int32)
    val = rng.uniform(-1, 1, len(col)) / width
    val[rp[1:] - 1] = rng.uniform(1, 2, len(rp) - 1)
    return rp, col, val.astype(vt)


def _kernel(kind, rp, col, val, b, k=1, row_major=True, mode=0):
    from smaxkernels_b200 import FloatType, Interface, IntType, KernelType, PlatformType
    n = len(rp) - 1
    smax = Interface()
    smax.register_kernel("t", KernelType[kind], PlatformType.CUDA, IntType.INT32,
                         FloatType.FLOAT64 if val.dtype == np.float64 else FloatType.FLOAT32)
    kern = smax.kernel("t")
    kern.set_solve_mode(mode)
    kern.set_mat_lower_triang(True)
    x = np.full(n * k, 7, val.dtype)
    dims = (n,) if kind == "SPTRSV" else (n, k)
    if kind == "SPTRSM":
        kern.set_vec_row_major(row_major)
    kern.register_A(n, n, len(col), col.copy(), rp, val.copy())
    kern.register_B(*dims, x)
    kern.register_C(*dims, b)
    return smax, kern, x


def _solve(*args, **kw):
    smax, kern, x = _kernel(*args, **kw)
    kern.run()
    smax.close()
    return x


MERGED = 2
EDGES = [1, 2, 3, 4, 5, 31, 33, 127, 128, 129, 1, 255, 256, 257, 479, 480, 481, 607, 608, 609, 1215, 1217, 2000, 7]


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("width", [1, 2, 3, 4, 9, 40])
@pytest.mark.parametrize("sizes", ["edges", "narrow", "wide"])
def test_sweep_vs_oracle(vt, width, sizes):
    sizes = {"edges": EDGES, "narrow": [5, 9, 1, 30] * 60, "wide": [700, 4097, 3, 4096, 50] * 2}[sizes]
    rp, col, val = level_matrix(sizes, width, width, vt)
    b = np.random.default_rng(1).uniform(-1, 1, len(rp) - 1).astype(vt)
    x = _solve("SPTRSV", rp, col, val, b)
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("width", [4, 5, 9, 40, 200])
@pytest.mark.parametrize("merge", [0, 4096])
def test_longer_rows_on_a_grid_and_in_runs(vt, width, merge):
    """Levels at the edges of a run's chunks, of a grid's CTAs and of the entries it takes at a time."""
    rp, col, val = level_matrix([3, 63, 64, 65, 1, 255, 257, 700, 31, 33, 128, 129] * 2, width, width, vt)
    n = len(rp) - 1
    b = np.random.default_rng(1).uniform(-1, 1, n).astype(vt)
    smax, kern, x = _kernel("SPTRSV", rp, col, val, b)
    kern.set_level_merge(merge)
    kern.run()
    smax.close()
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("width,sizes,k", [(12, [300] * 30, 3), (12, [300] * 30, 40), (40, [200] * 40, 3), (17, [64, 65, 2] * 20, 5)])
def test_blocks_of_longer_rows_equal_the_level_launches(vt, width, sizes, k):
    """Sweeps, with wide levels of several vectors, and what takes their place."""
    rp, col, val = level_matrix(sizes, width, 5, vt)
    b = np.random.default_rng(k).uniform(-1, 1, (len(rp) - 1) * k).astype(vt)
    for row_major in (True, False):
        x = _solve("SPTRSM", rp, col, val, b, k=k, row_major=row_major)
        np.testing.assert_array_equal(x, _solve("SPTRSM", rp, col, val, b, k=k, row_major=row_major, mode=MERGED))


@pytest.mark.parametrize("vt", [np.float64, np.float32])
def test_sweep_reads_solutions_older_than_the_ring(vt):
    """Recent and old sources mixed: 30000 rows against a ring of 8192."""
    rp, col, val = level_matrix([600] * 50, 4, 3, vt)
    b = np.random.default_rng(2).uniform(-1, 1, len(rp) - 1).astype(vt)
    x = _solve("SPTRSV", rp, col, val, b)
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("side", [96, 700])
def test_sweep_of_many_records_repeats(vt, side):
    """5-point lower triangle in natural order: enough records for the copies
    to go round the stage and their mbarriers many times; every solve is equal."""
    n = side * side
    r = np.arange(n)
    cols = np.stack([np.where(r >= side, r - side, -1), np.where(r % side, r - 1, -1), r], 1)
    keep = cols >= 0
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    col = cols[keep].astype(np.int32)
    rng = np.random.default_rng(side)
    val = (rng.uniform(-1, 1, len(col)) / 4).astype(vt)
    val[rp[1:] - 1] = rng.uniform(1, 2, n)
    b = rng.uniform(-1, 1, n).astype(vt)
    smax, kern, x = _kernel("SPTRSV", rp, col, val, b)
    kern.run()
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)
    first = x.copy()
    for _ in range(20):
        x[:] = 7
        kern.run()
        np.testing.assert_array_equal(x, first)
    smax.close()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
def test_sweep_rows_too_wide_for_the_stage(vt):
    """A row of 8000 entries among short ones is read in place."""
    rng = np.random.default_rng(4)
    n = 9000
    rows = [[r - 1, r] if r else [0] for r in range(n)]
    rows[8500] = list(range(500, 8500)) + [8500]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    val = (rng.uniform(-1, 1, len(col)) / 50).astype(vt)
    val[rp[1:] - 1] = rng.uniform(1, 2, n)
    b = rng.uniform(-1, 1, n).astype(vt)
    x = _solve("SPTRSV", rp, col, val, b)
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)


def test_sweep_waits_for_a_very_long_row():
    """A row of 400000 entries, read in place by one thread while the others
    wait for its level: as long as it takes."""
    n0, chain = 400000, 60
    n = n0 + 1 + chain
    rows = [np.array([r]) for r in range(n0)] + [np.arange(n0 + 1)] + [np.array([r - 1, r]) for r in range(n0 + 1, n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    rng = np.random.default_rng(11)
    val = rng.uniform(-1, 1, len(col)) / 1000
    val[rp[1:] - 1] = rng.uniform(1, 2, n)
    b = rng.uniform(-1, 1, n)
    x = _solve("SPTRSV", rp, col, val, b)
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(np.float64)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [2, 31, 33, 150])
@pytest.mark.parametrize("row_major", [True, False])
def test_blocks_equal_the_level_launches(vt, k, row_major):
    rp, col, val = level_matrix(EDGES, 3, 5, vt)
    b = np.random.default_rng(k).uniform(-1, 1, (len(rp) - 1) * k).astype(vt)
    x = _solve("SPTRSM", rp, col, val, b, k=k, row_major=row_major)
    np.testing.assert_array_equal(x, _solve("SPTRSM", rp, col, val, b, k=k, row_major=row_major, mode=MERGED))


@pytest.mark.parametrize("kind,k", [("SPTRSV", 1), ("SPTRSM", 5)])
def test_new_values_equal_a_new_kernel(kind, k):
    rp, col, val = level_matrix([40, 300, 5, 700] * 5, 5, 6, np.float64)
    n = len(rp) - 1
    rng = np.random.default_rng(7)
    b = rng.uniform(-1, 1, n * k)
    smax, kern, x = _kernel(kind, rp, col, val, b, k=k)
    kern.run()
    for _ in range(2):
        val = val * rng.uniform(0.5, 1.5, len(val))
        kern.update_A_values(val)
        kern.run()
        np.testing.assert_array_equal(x, _solve(kind, rp, col, val, b, k=k))
    smax.close()


def test_new_values_sync_free():
    """The sync-free pack (few wide levels) takes new values over as well."""
    rp, col, val = level_matrix([70000, 70000], 2, 8, np.float64)
    rng = np.random.default_rng(9)
    b = rng.uniform(-1, 1, len(rp) - 1)
    smax, kern, x = _kernel("SPTRSV", rp, col, val, b, mode=5)
    kern.run()
    val = val * rng.uniform(0.5, 1.5, len(val))
    kern.update_A_values(val)
    kern.run()
    np.testing.assert_array_equal(x, _solve("SPTRSV", rp, col, val, b, mode=5))
    smax.close()


def wide_levels(sizes, width, seed, vt):
    """level_matrix with exactly `width` sources a row, all in the level before."""
    rng = np.random.default_rng(seed)
    starts = np.concatenate([[0], np.cumsum(sizes)])
    cols, lens = [], []
    for s, m in enumerate(sizes):
        r = np.arange(starts[s], starts[s + 1])[:, None]
        c = rng.integers(starts[s - 1], starts[s], (m, width)) if s else np.zeros((m, 0), np.int64)
        cols.append(np.concatenate([c, r], 1).ravel())
        lens.append(np.full(m, c.shape[1] + 1))
    rp = np.concatenate([[0], np.cumsum(np.concatenate(lens))]).astype(np.int32)
    val = rng.uniform(-1, 1, rp[-1]) / width
    val[rp[1:] - 1] = rng.uniform(1, 2, len(rp) - 1)
    return rp, np.concatenate(cols).astype(np.int32), val.astype(vt)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("width", [1, 3, 5, 23])
@pytest.mark.parametrize("sizes", [[8188, 8189, 8192, 8193] * 5, [20000, 8500, 300, 9001, 16390] * 4])
def test_levels_wider_than_the_ring(vt, width, sizes):
    """Swept in one run, such a level writes some slots of the ring twice."""
    rp, col, val = wide_levels(sizes, width, width, vt)
    b = np.random.default_rng(width).uniform(-1, 1, len(rp) - 1).astype(vt)
    smax, kern, x = _kernel("SPTRSV", rp, col, val, b)
    kern.set_level_merge(1 << 20)
    kern.run()
    assert normwise(x, O.sptrsv(rp, col, val, b)) <= tol(vt)
    first = x.copy()
    for _ in range(10):
        kern.run()
        np.testing.assert_array_equal(x, first)
    smax.close()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
@pytest.mark.parametrize("count,most", [(3, 900), (170, 60)])
def test_batches(vt, count, most):
    """Few matrices with wide levels, and more matrices than SMs."""
    import torch
    from smaxkernels_b200.interface import FloatType, TriangularBatch
    rng = np.random.default_rng(count)
    mats = [level_matrix(rng.integers(1, most, 12).tolist(), 1 + m % 4, m, vt) for m in range(count)]
    tb = TriangularBatch(mats, FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    n = sum(len(m[0]) - 1 for m in mats)
    b = rng.uniform(-1, 1, n).astype(vt)
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    tb.solve(bd, xd)
    torch.cuda.synchronize()
    x = xd.cpu().numpy()
    for m, (rp, col, val) in enumerate(mats):
        a, e = tb.row_offset(m), tb.row_offset(m + 1)
        assert normwise(x[a:e], O.sptrsv(rp, col, val, b[a:e])) <= tol(vt), m
    tb.close()


@pytest.mark.parametrize("mode", [0, MERGED])
def test_a_wait_that_runs_out_in_a_batch_is_reported(mode):
    """solve() is asynchronous: sync() raises TIMEOUT, or else the next solve() does."""
    import torch
    from smaxkernels_b200 import SmaxError, _lib
    from smaxkernels_b200.interface import TriangularBatch
    rng = np.random.default_rng(13)
    mats = [level_matrix([40, 3, 90] * 6, 3, m, np.float64) for m in range(200)]
    tb = TriangularBatch(mats)
    b = rng.uniform(-1, 1, sum(len(m[0]) - 1 for m in mats))
    bd, xd = torch.from_numpy(b).cuda(), torch.zeros(len(b), dtype=torch.float64, device="cuda")
    tb._flag("spin_limit", 5)
    tb._flag("test_force_timeout", 1)
    for report in (tb.sync, lambda: (torch.cuda.synchronize(), tb.solve(bd, xd, mode))):
        tb.solve(bd, xd, mode)
        with pytest.raises(SmaxError) as e:
            report()
        assert e.value.code == _lib.ERR_TIMEOUT
        assert torch.isnan(xd).all()
    tb._flag("test_force_timeout", 0)
    tb.solve(bd, xd, mode)
    tb.sync()
    x = xd.cpu().numpy()
    for m, (rp, col, val) in enumerate(mats):
        a, e = tb.row_offset(m), tb.row_offset(m + 1)
        assert normwise(x[a:e], O.sptrsv(rp, col, val, b[a:e])) <= tol(np.float64), m
    tb.close()


@pytest.mark.parametrize("kind,k,mode", [("SPTRSV", 1, 0), ("SPTRSV", 1, MERGED), ("SPTRSM", 3, 0)])
@pytest.mark.parametrize("most", [30, 60, 400])
def test_a_wait_that_runs_out_is_an_error_and_recoverable(kind, k, mode, most):
    """A level waits for an arrival that never comes: the sweep ends, reports
    TIMEOUT and leaves no number behind, and the same kernel solves afterwards."""
    from smaxkernels_b200 import SmaxError, _lib
    rp, col, val = level_matrix([most, most - 3, 2] * 20, 4, most, np.float64)
    n = len(rp) - 1
    b = np.random.default_rng(12).uniform(-1, 1, n * k)
    smax, kern, x = _kernel(kind, rp, col, val, b, k=k, mode=mode)
    kern.set_spin_limit(5)
    kern._flag("test_force_timeout", 1)
    with pytest.raises(SmaxError) as e:
        kern.run()
    assert e.value.code == _lib.ERR_TIMEOUT
    assert np.isnan(x).all()
    kern._flag("test_force_timeout", 0)
    kern.run()
    smax.close()
    B = b.reshape(n, k)
    ref = np.stack([O.sptrsv(rp, col, val, np.ascontiguousarray(B[:, v])) for v in range(k)], 1)
    assert normwise(x.reshape(n, k), ref) <= tol(np.float64)


@pytest.mark.parametrize("vt", [np.float64, np.float32])
def test_batch_of_more_matrices_than_sms_with_narrow_levels(vt):
    """Levels of at most 30 rows: two CTAs share an SM and half the stage each, and
    take several matrices one after the other; some of one row, one with a row
    of 300 entries, which that stage does not hold."""
    import torch
    from smaxkernels_b200.interface import FloatType, TriangularBatch
    rng = np.random.default_rng(4)
    count = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 104
    mats = [level_matrix([1] if m % 50 == 7 else rng.integers(1, 31, 12).tolist(), 1 + m % 5, m, vt) for m in range(count)]
    n = 400
    rows = [[r - 1, r] if r else [0] for r in range(n)]
    rows[350] = list(range(50, 350)) + [350]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    val = rng.uniform(-1, 1, rp[-1]) / 20
    val[rp[1:] - 1] = rng.uniform(1, 2, n)
    mats[100] = (rp, np.concatenate(rows).astype(np.int32), val.astype(vt))
    tb = TriangularBatch(mats, FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    b = rng.uniform(-1, 1, sum(len(m[0]) - 1 for m in mats)).astype(vt)
    bd = torch.from_numpy(b).cuda()
    xd, again = torch.zeros_like(bd), torch.zeros_like(bd)
    tb.solve(bd, xd)
    tb.solve(bd, again)
    tb.sync()
    assert torch.equal(xd, again)
    x = xd.cpu().numpy()
    for m, (rp, col, val) in enumerate(mats):
        a, e = tb.row_offset(m), tb.row_offset(m + 1)
        assert normwise(x[a:e], O.sptrsv(rp, col, val, b[a:e])) <= tol(vt), m
    tb.close()


@pytest.mark.parametrize("vt", [np.float64, np.float32])
def test_batches_with_levels_for_the_whole_chip(vt):
    """Few matrices of wide levels, of different depth, one without levels to wait for."""
    import torch
    from smaxkernels_b200.interface import FloatType, TriangularBatch
    mats = [wide_levels([9000] * 6, 3, 1, vt), wide_levels([20000, 1], 5, 2, vt), wide_levels([5], 1, 3, vt),
            wide_levels([3000] * 9, 8, 4, vt)]
    tb = TriangularBatch(mats, FloatType.FLOAT64 if vt == np.float64 else FloatType.FLOAT32)
    b = np.random.default_rng(3).uniform(-1, 1, sum(len(m[0]) - 1 for m in mats)).astype(vt)
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    for mode in (0, MERGED):
        xd.zero_()
        tb.solve(bd, xd, mode)
        tb.sync()
        x = xd.cpu().numpy()
        for m, (rp, col, val) in enumerate(mats):
            a, e = tb.row_offset(m), tb.row_offset(m + 1)
            assert normwise(x[a:e], O.sptrsv(rp, col, val, b[a:e])) <= tol(vt), m
    tb.close()


def test_batch_of_a_level_with_more_chunks_than_a_barrier_counts():
    """One diagonal matrix of 2^18 chunks of 256 rows and a little more, and a small one."""
    import torch
    from smaxkernels_b200.interface import FloatType, TriangularBatch
    n = (1 << 26) + 3000
    d = (np.arange(n) % 7 + 1).astype(np.float32)
    small = level_matrix([3, 5], 2, 0, np.float32)
    tb = TriangularBatch([(np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d), small], FloatType.FLOAT32)
    b = torch.ones(n + 8, dtype=torch.float32, device="cuda")
    x = torch.zeros_like(b)
    tb.solve(b, x)
    tb.sync()
    assert torch.equal(x[:n], 1 / torch.from_numpy(d).cuda())
    assert normwise(x[n:].cpu().numpy(), O.sptrsv(*small, np.ones(8, np.float32))) <= tol(np.float32)
    tb.close()


def test_a_refused_merge_threshold_closes_no_other():
    """A level of 5200 rows of up to 43500 entries is too much for one run: the
    plain kernels solve with the threshold that would sweep it, and the pack, which
    multiplies by 1/D where they divide, with one that leaves it to a grid."""
    sources, m, tail = 45000, 5200, 2000
    rng = np.random.default_rng(14)
    lens = np.concatenate([[0, 0, 0], np.ones(sources), np.full(m, 14500), np.ones(tail)]).astype(np.int64)
    lens[3 + sources] = 43500
    n = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens + 1)]).astype(np.int32)
    col = np.empty(rp[-1], np.int32)
    col[rp[1:] - 1] = np.arange(n)
    off = np.ones(len(col), bool)
    off[rp[1:] - 1] = False
    wide = np.arange(rp[3 + sources], rp[3 + sources + m])
    col[rp[3]:rp[3 + sources]][::2] = rng.integers(0, 3, sources)
    w = wide[off[wide]]
    col[w] = 3 + (np.arange(len(w)) * 7 + np.arange(len(w)) // sources) % sources
    t0 = 3 + sources + m
    col[rp[t0]:][::2] = np.arange(t0 - 1, n - 1)
    val = rng.uniform(-1, 1, len(col)).astype(np.float32) / 1000
    val[rp[1:] - 1] = rng.uniform(1, 2, n)
    b = rng.uniform(-1, 1, n).astype(np.float32)
    fresh = _solve("SPTRSV", rp, col, val, b)
    smax, kern, x = _kernel("SPTRSV", rp, col, val, b)
    kern.set_level_merge(1 << 20)
    kern.run()
    assert normwise(x, fresh) <= tol(np.float32) and not np.array_equal(x, fresh)
    kern.set_level_merge(4096)
    kern.run()
    np.testing.assert_array_equal(x, fresh)
    smax.close()
