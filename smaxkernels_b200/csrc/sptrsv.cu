// sptrsv.cu -- level-scheduled SpTRSV / SpTRSM on sm_100a.
//
// Reference semantics:
//   * peel_diag_crs (src/kernels/sptrsv/sptrsv_cpu/sptrsv_cpu_crs_helpers_impl.hpp:9-38):
//     D[r] = A[r][r] (the last diagonal entry of the row), swapped to the last
//     slot of its row; |D| < 1e-16 or a missing diagonal is an error.
//   * naive_crs_sptrsv / crs_sptrsv_lvl (sptrsv_cpu_crs_impl.hpp:9-55,
//     sptrsv_lvl_cpu_crs_impl.hpp:11-82) and the SpTRSM loops
//     (src/kernels/sptrsm/sptrsm_cpu/sptrsm_cpu_crs_impl.hpp:9-102):
//     x[r] = (b[r] - sum_{j < end-1} val[j] x[col[j]]) / D[r].
//
// Schedule.  A solve is a sequence of levels; the rows of one level are
// independent.  With the permuted (level-scheduled) flag the levels are the
// caller's contiguous row ranges (generate_perm's lvl_ptr), swept ascending for
// lower and descending for upper triangles, as the reference does.  Without
// it the platform computes the dependency levels of the matrix itself
// (levels.cu: RS levels of A+A^T, reversed for upper triangles) and keeps a
// row order, so the plain solve runs level-parallel with the reference's
// per-row arithmetic and summation order.
//
// Kernels.  One thread per (row, right-hand side) sums its row sequentially.
//   * wide level: one grid launch per level;
//   * run of narrow levels (<= merge threshold rows * k each): one CTA sweeps
//     the whole run, with __syncthreads() as the level barrier (global writes
//     of the CTA are visible to the CTA after the barrier);
// The launch sequence of a solve can be captured once into a CUDA graph and
// replayed (tri_solve_graph).
#include "sptrsv.cuh"

#include <algorithm>

namespace smax {

namespace {

constexpr int kSegThreads = 1024;

// ------------------------------------------------------------ peel diag ----
template <typename VT>
__global__ void peel_diag_kernel(const int *__restrict__ rp, int *__restrict__ col, VT *__restrict__ val, int64_t n,
                                 VT *__restrict__ D, DevStatus *st) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int s = rp[r], e = rp[r + 1] - 1;
    int dj = -1;
    for (int j = s; j <= e; ++j)
        if (col[j] == (int)r) dj = j;  // the last diagonal entry wins, as in the reference
    if (dj < 0) {
        report(st, SMAX_ERR_NO_DIAG, r);
        return;
    }
    const VT d = val[dj];
    if (fabs((double)d) < 1e-16) report(st, SMAX_ERR_ZERO_DIAG, r);
    D[r] = d;
    if (dj != e) {
        const int tc = col[dj];
        col[dj] = col[e];
        col[e] = tc;
        const VT tv = val[dj];
        val[dj] = val[e];
        val[e] = tv;
    }
}

// D[r] = the last entry of row r, which the peel made the diagonal
template <typename VT>
__global__ void refresh_diag_kernel(const int *__restrict__ rp, const int *__restrict__ col,
                                    const VT *__restrict__ val, int64_t n, VT *__restrict__ D, DevStatus *st) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int e = rp[r + 1] - 1;
    if (e < rp[r] || col[e] != (int)r) {
        report(st, SMAX_ERR_NO_DIAG, r);
        return;
    }
    const VT d = val[e];
    if (fabs((double)d) < 1e-16) report(st, SMAX_ERR_ZERO_DIAG, r);
    D[r] = d;
}

// ------------------------------------------------------------ the row op ---
// Element (row r, vector v) of X / B lives at r*rs + v*vs.
template <typename VT>
__device__ __forceinline__ void solve_row(const int *__restrict__ rp, const int *__restrict__ col,
                                          const VT *__restrict__ val, const VT *__restrict__ D, const VT *B, VT *X,
                                          int r, int64_t v, int64_t rs, int64_t vs) {
    const int s = rp[r], e = rp[r + 1] - 1;  // the diagonal sits at e
    VT sum = VT(0);
    const int64_t vo = v * vs;
    for (int j = s; j < e; ++j) sum += val[j] * X[(int64_t)col[j] * rs + vo];
    X[(int64_t)r * rs + vo] = (B[(int64_t)r * rs + vo] - sum) / D[r];
}

// thread t -> (i-th row of the level, vector v); rows vary fastest for
// column-major blocks, vectors for row-major ones (coalesced X accesses)
__device__ __forceinline__ void split_work(int64_t t, int64_t m, int64_t k, bool row_major, int64_t &i,
                                           int64_t &v) {
    if (row_major) { i = t / k; v = t % k; }
    else { i = t % m; v = t / m; }
}

template <typename VT>
__global__ void level_kernel(const int *__restrict__ rp, const int *__restrict__ col, const VT *__restrict__ val,
                             const VT *__restrict__ D, const int *__restrict__ order, int row0, int m, int64_t k,
                             bool row_major, int64_t rs, int64_t vs, const VT *B, VT *X) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)m * k) return;
    int64_t i, v;
    split_work(t, m, k, row_major, i, v);
    const int r = order ? order[row0 + i] : row0 + (int)i;
    solve_row<VT>(rp, col, val, D, B, X, r, v, rs, vs);
}

// One CTA sweeps levels seg_lvl[0..n_lvls) (given as [begin, end) row ranges
// into `order`, or contiguous rows when order is null).
template <typename VT>
__global__ void __launch_bounds__(kSegThreads) segment_kernel(const int *__restrict__ rp, const int *__restrict__ col,
                                                              const VT *__restrict__ val, const VT *__restrict__ D,
                                                              const int *__restrict__ order,
                                                              const int2 *__restrict__ ranges, int n_lvls, int64_t k,
                                                              bool row_major, int64_t rs, int64_t vs, const VT *B,
                                                              VT *X) {
    for (int l = 0; l < n_lvls; ++l) {
        const int2 rg = ranges[l];
        const int64_t m = rg.y - rg.x;
        for (int64_t t = threadIdx.x; t < m * k; t += blockDim.x) {
            int64_t i, v;
            split_work(t, m, k, row_major, i, v);
            const int r = order ? order[rg.x + i] : rg.x + (int)i;
            solve_row<VT>(rp, col, val, D, B, X, r, v, rs, vs);
        }
        __syncthreads();
    }
}

}  // namespace

void peel_diag(DevCRS &a, int vbytes, DevBuf &D, DevStatus *st, cudaStream_t s) {
    D.alloc((size_t)vbytes * (a.n_rows ? a.n_rows : 1));
    if (a.n_rows == 0) return;
    const unsigned g = ceil_div_u(a.n_rows, 256);
    if (vbytes == 8)
        peel_diag_kernel<double><<<g, 256, 0, s>>>(a.rp(), a.col.as<int>(), a.val.as<double>(), a.n_rows,
                                                   D.as<double>(), st);
    else
        peel_diag_kernel<float><<<g, 256, 0, s>>>(a.rp(), a.col.as<int>(), a.val.as<float>(), a.n_rows,
                                                  D.as<float>(), st);
    SMAX_CUDA(cudaGetLastError());
}

void refresh_diag(const DevCRS &a, int vbytes, DevBuf &D, DevStatus *st, cudaStream_t s) {
    if (a.n_rows == 0) return;
    const unsigned g = ceil_div_u(a.n_rows, 256);
    if (vbytes == 8)
        refresh_diag_kernel<double><<<g, 256, 0, s>>>(a.rp(), a.ci(), a.val.as<double>(), a.n_rows, D.as<double>(), st);
    else
        refresh_diag_kernel<float><<<g, 256, 0, s>>>(a.rp(), a.ci(), a.val.as<float>(), a.n_rows, D.as<float>(), st);
    SMAX_CUDA(cudaGetLastError());
}

void TriPlan::build_own(const DevCRS &a, bool upper, cudaStream_t st) {
    DevBuf srp, scol, lvl;
    int64_t snnz = 0;
    build_symmetric(a, srp, scol, snnz, st);
    const int nl = rs_levels(srp.as<int>(), scol.as<int>(), a.n_rows, lvl, st, upper);
    level_order(lvl.as<int>(), a.n_rows, nl, order, lvl_ptr, st);
    if (a.n_rows > 0 && lvl_ptr.back() != a.n_rows) fail(SMAX_ERR_STATE, "dependency levels do not cover all rows");
    has_order = true;
    descending = false;
    n_rows = a.n_rows;
    finish(st);
}

void TriPlan::build_given(const std::vector<int> &lp, int64_t n, bool upper, cudaStream_t st) {
    if (lp.empty() || lp.front() != 0 || lp.back() != n) fail(SMAX_ERR_STATE, "level pointer does not match the matrix");
    for (size_t i = 1; i < lp.size(); ++i)
        if (lp[i] < lp[i - 1]) fail(SMAX_ERR_BAD_ARG, "level pointer is not monotone");
    lvl_ptr = lp;
    order.release();
    has_order = false;
    descending = upper;  // crs_sptrsv_lvl<false> walks levels from last to first
    n_rows = n;
    finish(st);
}

void TriPlan::assign_reverse(const TriPlan &src, cudaStream_t st) {
    release_graph();
    n_rows = src.n_rows;
    lvl_ptr = src.lvl_ptr;
    has_order = src.has_order;
    descending = !src.descending;
    if (src.has_order) {
        order.alloc(sizeof(int) * (n_rows > 0 ? n_rows : 1));
        if (n_rows) SMAX_CUDA(cudaMemcpyAsync(order.p, src.order.p, sizeof(int) * n_rows, cudaMemcpyDeviceToDevice, st));
    } else {
        order.release();
    }
    scheduled_k = -1;
    scheduled_merge = -1;
    finish(st);
}

void TriPlan::finish(cudaStream_t) {
    graph_valid = false;
    pack_ok = false;
    pack_refused.clear();
    pack = SweepPack();
    sf_ok = false;
    sf_unfit = false;
    sf_pack = LevelPack();
}

bool TriPlan::ensure_pack(const int *rp, const int *ci, const void *val, const void *D, int vbytes, int merge_rows,
                          uint64_t tag, cudaStream_t st, int64_t k) {
    merge_rows = run_threshold(merge_rows);
    if (pack_unfit(merge_rows, k)) return false;
    if (!pack_is(val, D, vbytes, merge_rows, pack_tag, k)) {
        if (scheduled_k != 1 || scheduled_merge != merge_rows) schedule(1, merge_rows);
        const int L = n_levels();
        std::vector<int> src_begin(L), count(L);
        std::vector<SweepStep> sweep;
        for (const Step &s : steps) {
            for (int i = 0; i < s.sweep_count; ++i) {
                const int sw = s.sweep_first + i;
                const int lv = descending ? L - 1 - sw : sw;
                src_begin[sw] = lvl_ptr[lv];
                count[sw] = lvl_ptr[lv + 1] - lvl_ptr[lv];
            }
            sweep.push_back(SweepStep{s.sweep_first, s.sweep_count, s.kind});
        }
        release_graph();
        ++pack_serial;
        pack_ok = false;
        const bool ok = build_sweep_pack(pack, rp, ci, val, D, vbytes, n_rows, has_order ? order.as<int>() : nullptr,
                                         src_begin, count, sweep, k > 1, false, st);
        if (!ok) {
            pack_refused.push_back({merge_rows, k > 1});
            return false;
        }
        pack_ok = true;
        pack_key[0] = val;
        pack_key[1] = D;
        pack_tag = tag;
        pack_merge = merge_rows;
        pack_vbytes = vbytes;
    } else if (pack_tag != tag) {
        // new values on the same pattern: in place, so a captured graph stays valid
        refill_sweep_pack(pack, rp, val, D, st);
        pack_tag = tag;
    }
    const void *before[2] = {pack.bp.p, pack.xp.p};
    const int vectors = pack.vectors;
    sweep_reserve(pack, k);
    if (pack.bp.p != before[0] || pack.xp.p != before[1] || pack.vectors != vectors) {
        release_graph();
        ++pack_serial;
    }
    return true;
}

bool TriPlan::ensure_syncfree(const int *rp, const int *ci, const void *val, const void *D, int vbytes, uint64_t tag,
                              bool values, cudaStream_t st) {
    if (sf_ok && sf_key[0] == val && sf_key[1] == D && sf_vbytes == vbytes) {
        if (values && sf_tag != tag) {
            refill_level_pack(sf_pack, rp, val, D, st);
            sf_tag = tag;
        }
        return true;
    }
    if (sf_unfit) return false;  // a property of the pattern and the level sets
    const int L = n_levels();
    std::vector<int> src_begin(L), count(L);
    for (int sw = 0; sw < L; ++sw) {
        const int lv = descending ? L - 1 - sw : sw;
        src_begin[sw] = lvl_ptr[lv];
        count[sw] = lvl_ptr[lv + 1] - lvl_ptr[lv];
    }
    sf_ok = false;
    const bool ok = build_level_pack(sf_pack, rp, ci, val, D, vbytes, n_rows, has_order ? order.as<int>() : nullptr,
                                     src_begin, count, st);
    if (!ok || sf_pack.reads_unsolved) {
        sf_pack = LevelPack();
        sf_unfit = true;
        return false;
    }
    sf_ok = true;
    sf_key[0] = val;
    sf_key[1] = D;
    sf_tag = tag;
    sf_vbytes = vbytes;
    return true;
}

void TriPlan::prepare(int64_t k, int merge_rows, cudaStream_t st) {
    if (scheduled_k != k || scheduled_merge != merge_rows) schedule(k, merge_rows);
    if (!ranges_uploaded && !seg_ranges.empty()) {
        SMAX_CUDA(cudaMemcpyAsync(d_ranges.p, seg_ranges.data(), sizeof(int2) * seg_ranges.size(),
                                  cudaMemcpyHostToDevice, st));
        ranges_uploaded = true;
        SMAX_CUDA(cudaStreamSynchronize(st));
    }
}

// Up to kLeadLevels levels of more than kRunStart rows at the start of a run
// are launches of their own: their sources are wide levels and rows long
// solved, which the sweep would read from global memory, and a launch is the
// faster way through such a level then (a longer row of wide levels is a band,
// with its sources in the ring).  Rows ordered by level sets, FP64, 200^2:
// 40.5 us; with 1024 rows 42.9, 2048 48.5, no limit 59.0.
constexpr int kLeadLevels = 16;
constexpr int64_t kRunStart = 512;

// Sequence of steps: wide levels alone, runs of narrow levels merged.
void TriPlan::schedule(int64_t k, int merge_rows) {
    steps.clear();
    seg_ranges.clear();
    const int L = (int)lvl_ptr.size() - 1;
    int l = 0;
    auto level_at = [&](int idx) { return descending ? L - 1 - idx : idx; };
    auto level_rows = [&](int idx) {
        const int lv = level_at(idx);
        return (int64_t)(lvl_ptr[lv + 1] - lvl_ptr[lv]);
    };
    while (l < L) {
        const int lv = level_at(l);
        const int64_t m = level_rows(l);
        int end = l;
        while (end < L && merge_rows > 0 && level_rows(end) * k <= merge_rows) ++end;
        if (k == 1) {
            int lead = l;
            while (lead < end && lead - l <= kLeadLevels && level_rows(lead) > kRunStart) ++lead;
            if (lead > l && lead - l <= kLeadLevels) end = l;
        }
        if (end > l) {
            // one run: splitting it by width, with fewer threads for the
            // narrower stretches, measured slower (FP64 5-point D+L, 512^2 in
            // natural order: 271 us in three runs, 260 us in one)
            Step s;
            s.kind = 1;
            s.seg_first = (int)seg_ranges.size();
            s.sweep_first = l;
            for (; l < end; ++l) {
                const int lv2 = level_at(l);
                seg_ranges.push_back({lvl_ptr[lv2], lvl_ptr[lv2 + 1]});
            }
            s.seg_count = (int)seg_ranges.size() - s.seg_first;
            s.sweep_count = s.seg_count;
            steps.push_back(s);
        } else {
            Step s;
            s.kind = 0;
            s.row0 = lvl_ptr[lv];
            s.m = (int)m;
            s.sweep_first = l;
            s.sweep_count = 1;
            steps.push_back(s);
            ++l;
        }
    }
    d_ranges.alloc(sizeof(int2) * (seg_ranges.empty() ? 1 : seg_ranges.size()));
    scheduled_k = k;
    scheduled_merge = merge_rows;
    ranges_uploaded = false;
    graph_valid = false;
}

template <typename VT>
void tri_solve(TriPlan &p, const DevCRS &a, const VT *D, const VT *B, VT *X, int64_t k, bool row_major, int64_t ld,
               int merge_rows, uint64_t tag, cudaStream_t st) {
    if (k == 1 && p.n_rows > 0) p.ensure_pack(a.rp(), a.ci(), a.val.p, D, sizeof(VT), merge_rows, tag, st);
    tri_solve_raw<VT>(p, a.rp(), a.ci(), a.val.as<VT>(), D, B, X, k, row_major, ld, merge_rows, tag, st);
}

template <typename VT>
void tri_solve_raw(TriPlan &p, const int *rp, const int *ci, const VT *val, const VT *D, const VT *B, VT *X,
                   int64_t k, bool row_major, int64_t ld, int merge_rows, uint64_t tag, cudaStream_t st) {
    if (p.n_rows == 0) return;
    const int64_t rs = row_major ? k : 1, vs = row_major ? 1 : ld;
    if (k == 1 && p.pack_is(val, D, sizeof(VT), merge_rows, tag, 1)) {
        sweep_solve<VT>(p.pack, B, X, 1, rs, vs, p.status, p.wait, st);
        return;
    }
    if (p.scheduled_k != k || p.scheduled_merge != merge_rows) p.schedule(k, merge_rows);
    if (!p.ranges_uploaded && !p.seg_ranges.empty()) {
        SMAX_CUDA(cudaMemcpyAsync(p.d_ranges.p, p.seg_ranges.data(), sizeof(int2) * p.seg_ranges.size(),
                                  cudaMemcpyHostToDevice, st));
        p.ranges_uploaded = true;
    }
    const int *order = p.has_order ? p.order.as<int>() : nullptr;
    const int2 *ranges = p.d_ranges.as<int2>();
    for (const auto &s : p.steps) {
        if (s.kind == 0) {
            const int64_t work = (int64_t)s.m * k;
            level_kernel<VT><<<ceil_div_u(work, 256), 256, 0, st>>>(rp, ci, val, D, order, s.row0, s.m, k, row_major,
                                                                    rs, vs, B, X);
        } else {
            segment_kernel<VT><<<1, kSegThreads, 0, st>>>(rp, ci, val, D, order, ranges + s.seg_first, s.seg_count, k,
                                                          row_major, rs, vs, B, X);
        }
    }
    SMAX_CUDA(cudaGetLastError());
}

template <typename VT>
void tri_solve_graph(TriPlan &p, const DevCRS &a, const VT *D, const VT *B, VT *X, int64_t k, bool row_major,
                     int64_t ld, int merge_rows, uint64_t tag, cudaStream_t caller) {
    if (p.n_rows == 0) return;
    // the pack is built outside the capture (it synchronises); a rebuild drops the graph
    bool packed = false;
    if (k == 1 || sweep_suits(p, k, merge_rows)) {
        try {
            packed = p.ensure_pack(a.rp(), a.ci(), a.val.p, D, sizeof(VT), merge_rows, tag, caller, k);
        } catch (const Error &e) {
            // a block without room for the pack, or for the workspace of one vector,
            // runs the level launches, now and later
            if (k == 1 || e.code != SMAX_ERR_OOM) throw;
            p.pack = SweepPack();
            p.pack_ok = false;
            p.pack_refused.push_back({p.run_threshold(merge_rows), true});
            p.release_graph();
        }
    }
    // graphs are captured (and replayed) on a capturable stream
    const bool fenced = !is_capturable(caller);
    cudaStream_t st = fenced ? p.aux.enter(caller) : caller;
    struct Leave {
        TriPlan &p;
        bool fenced;
        cudaStream_t caller;
        ~Leave() {
            if (fenced) {
                cudaEventRecord(p.aux.out, p.aux.s);
                cudaStreamWaitEvent(caller, p.aux.out, 0);
            }
        }
    } leave{p, fenced, caller};
    if (!packed && (p.scheduled_k != k || p.scheduled_merge != merge_rows)) p.schedule(k, merge_rows);
    const void *key[4] = {B, X, D, a.val.p};
    if (!p.graph_valid || p.graph_key[0] != key[0] || p.graph_key[1] != key[1] || p.graph_key[2] != key[2] ||
        p.graph_key[3] != key[3] || p.graph_row_major != row_major || p.graph_ld != ld || p.graph_k != k || p.graph_packed != packed ||
        p.graph_wait != p.wait) {
        if (!packed && !p.ranges_uploaded && !p.seg_ranges.empty()) {
            SMAX_CUDA(cudaMemcpyAsync(p.d_ranges.p, p.seg_ranges.data(), sizeof(int2) * p.seg_ranges.size(),
                                      cudaMemcpyHostToDevice, st));
            p.ranges_uploaded = true;
        }
        SMAX_CUDA(cudaStreamSynchronize(st));
        p.release_graph();
        cudaGraph_t g = nullptr;
        SMAX_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            if (packed)
                sweep_solve<VT>(p.pack, B, X, k, row_major ? k : 1, row_major ? 1 : ld, p.status, p.wait, st);
            else
                tri_solve_raw<VT>(p, a.rp(), a.ci(), a.val.as<VT>(), D, B, X, k, row_major, ld, merge_rows, tag, st);
        } catch (...) {
            cudaStreamEndCapture(st, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        SMAX_CUDA(cudaStreamEndCapture(st, &g));
        cudaGraphExec_t ge = nullptr;
        cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        cuda_check(e, "cudaGraphInstantiate");
        p.graph = ge;
        p.graph_valid = true;
        p.graph_key[0] = key[0];
        p.graph_key[1] = key[1];
        p.graph_key[2] = key[2];
        p.graph_key[3] = key[3];
        p.graph_row_major = row_major;
        p.graph_ld = ld;
        p.graph_k = k;
        p.graph_packed = packed;
        p.graph_wait = p.wait;
    }
    SMAX_CUDA(cudaGraphLaunch(p.graph, st));
}

void TriPlan::release_graph() {
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    graph_valid = false;
}

TriPlan::~TriPlan() { release_graph(); }

// One SM goes through a level of 4096 entries in about the time of a launch: 0.3 ns
// an entry whose solution is in the ring, 0.8 to 1.3 from global memory, against
// 2.3 us and a whole chip.  FP64, random sources, run / grid: 1500 rows of 3 entries 3.1 /
// 2.2 us a level, of 8 8.9 / 4.0, of 40 69 / 5.5; 600 of 8 3.9 / 3.7; 200 of 40 10 / 5.2; 30 of
// 40 3.6 / 4.8.  Rows of two entries (5-point triangles) stay in runs up to 4096.
int default_run_rows(int64_t n_rows, int64_t off_diag) {
    constexpr int kRows = 4096;
    if (2 * off_diag <= 5 * n_rows) return kRows;
    return (int)std::max<int64_t>(1, (int64_t)kRows * n_rows / off_diag);
}

// k > 1 vectors: the wide levels of the sweeps read a solution from k separate
// vectors, where the level launches and the sync-free rows read k neighbours.
// FP64, random sources, sweeps / those: 1500 x 40 levels of 3 entries k = 32 124 / 123 us, of 8 200
// / 136, k = 4 173 / 136, of 40 k = 32 422 / 272, k = 4 235 / 284; 600 x 60 of 8 k = 32 237 / 197, k = 4 236 / 456;
// 200 x 100 of 40 k = 32 530 / 635.
bool sweep_suits(const TriPlan &p, int64_t k, int merge_rows) {
    const int64_t L = p.n_levels();
    return L > 0 && !p.pack_unfit(merge_rows, 2) && p.n_rows <= L * 2048 &&
           (p.off_diag <= L * 4096 || p.n_rows * k <= L * 8192);
}

bool syncfree_suits(const TriPlan &p, int64_t k, int merge_rows) {
    const int64_t L = p.n_levels();
    if (L <= 0 || (k > 1 && sweep_suits(p, k, merge_rows))) return false;
    if (k == 1) return p.n_rows >= (1 << 17) && p.n_rows >= L * 32768;
    return p.n_rows >= (1 << 16) && L >= 64 && p.n_rows <= L * 16384;
}

template <typename VT>
bool tri_solve_syncfree(TriPlan &p, const DevCRS &a, const VT *D, const VT *B, VT *X, uint64_t tag, DevBuf &ctl,
                        long long limit, bool force_timeout, DevStatus *st, cudaStream_t s, int64_t k,
                        bool row_major) {
    if (p.n_rows == 0 || k == 0) return true;
    const uintptr_t b0 = reinterpret_cast<uintptr_t>(B), x0 = reinterpret_cast<uintptr_t>(X);
    const uintptr_t len = sizeof(VT) * (uintptr_t)p.n_rows * (uintptr_t)k;
    if (b0 < x0 + len && x0 < b0 + len) return false;  // B is read while X fills
    if (!p.ensure_syncfree(a.rp(), a.ci(), a.val.p, D, sizeof(VT), tag, k == 1, s)) return false;
    ctl.ensure(64);
    if (k == 1)
        pack_solve_syncfree<VT>(p.sf_pack, B, X, ctl.p, limit, force_timeout, st, s);
    else
        solve_syncfree_rows<VT>(p.sf_pack, a.rp(), a.ci(), a.val.as<VT>(), D, B, X, k, row_major, ctl.p, limit, st,
                                s);
    return true;
}

template bool tri_solve_syncfree<double>(TriPlan &, const DevCRS &, const double *, const double *, double *, uint64_t,
                                         DevBuf &, long long, bool, DevStatus *, cudaStream_t, int64_t, bool);
template bool tri_solve_syncfree<float>(TriPlan &, const DevCRS &, const float *, const float *, float *, uint64_t,
                                        DevBuf &, long long, bool, DevStatus *, cudaStream_t, int64_t, bool);
template void tri_solve<double>(TriPlan &, const DevCRS &, const double *, const double *, double *, int64_t, bool,
                                int64_t, int, uint64_t, cudaStream_t);
template void tri_solve<float>(TriPlan &, const DevCRS &, const float *, const float *, float *, int64_t, bool,
                               int64_t, int, uint64_t, cudaStream_t);
template void tri_solve_raw<double>(TriPlan &, const int *, const int *, const double *, const double *,
                                    const double *, double *, int64_t, bool, int64_t, int, uint64_t, cudaStream_t);
template void tri_solve_raw<float>(TriPlan &, const int *, const int *, const float *, const float *, const float *,
                                   float *, int64_t, bool, int64_t, int, uint64_t, cudaStream_t);
template void tri_solve_graph<double>(TriPlan &, const DevCRS &, const double *, const double *, double *, int64_t,
                                      bool, int64_t, int, uint64_t, cudaStream_t);
template void tri_solve_graph<float>(TriPlan &, const DevCRS &, const float *, const float *, float *, int64_t, bool,
                                     int64_t, int, uint64_t, cudaStream_t);

}  // namespace smax
