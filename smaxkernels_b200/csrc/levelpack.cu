// levelpack.cu -- sync-free triangular solves on level-ordered packs, sm_100a.
//
// The per-row recurrence is the reference's (naive_crs_sptrsv / crs_sptrsv_lvl,
// src/kernels/sptrsv/sptrsv_cpu/sptrsv_cpu_crs_impl.hpp:9-55,
// sptrsv_lvl_cpu_crs_impl.hpp:11-82): x[r] = (b[r] - sum_j val[j] x[col[j]]) / D[r]
// with the off-diagonal entries summed in stored order.  Rows are renumbered in
// sweep order and each level's off-diagonal entries are stored as a dense
// column-major block, so a thread finds its row's entries at a fixed offset:
// no row_ptr hop, coalesced loads.  One launch solves all levels, each row
// waiting for the values it reads (levelpack.cuh).
#include "levelpack.cuh"

#include <algorithm>

#include <cub/device/device_segmented_reduce.cuh>

namespace smax {

namespace {

using Level = LevelPack::Level;
constexpr int kPad = LevelPack::kPad;

unsigned grid_for(int64_t work) {
    const int64_t cap = (int64_t)sm_count() * 8;
    int64_t g = (work + 255) / 256;
    return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

// ---------------------------------------------------------------- build ----
__global__ void positions_kernel(const int *__restrict__ pos_begin, int n_lv, const int *__restrict__ src_begin,
                                 const int *__restrict__ order, int64_t n, int *__restrict__ prow,
                                 int *__restrict__ plev, int *__restrict__ pos_of_row) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        int lo = 0, hi = n_lv - 1;  // last s with pos_begin[s] <= p
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pos_begin[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        const int k = src_begin[lo] + (int)(p - pos_begin[lo]);
        const int r = order ? order[k] : k;
        prow[p] = r;
        plev[p] = lo;
        pos_of_row[r] = (int)p;
    }
}

__global__ void off_len_kernel(const int *__restrict__ rp, const int *__restrict__ prow, int64_t n,
                               int *__restrict__ len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        const int r = prow[p];
        len[p] = rp[r + 1] - rp[r] - 1;
    }
}

template <typename VT>
__global__ void fill_kernel(const int *__restrict__ rp, const int *__restrict__ ci, const VT *__restrict__ val,
                            const VT *__restrict__ D, int64_t n, const int *__restrict__ prow,
                            const int *__restrict__ plev, const int *__restrict__ pos_of_row,
                            const Level *__restrict__ lv, int *__restrict__ psrc, VT *__restrict__ pval,
                            VT *__restrict__ pinv, int *reads_unsolved) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        const Level L = lv[plev[p]];
        const int t = (int)(p - L.pos);
        const int r = prow[p];
        const int j0 = rp[r], len = rp[r + 1] - j0 - 1;
        for (int i = 0; i < L.w; ++i) {
            const long long idx = L.base + (long long)i * L.m + t;
            if (i < len) {
                const int c = ci[j0 + i];
                if (pos_of_row[c] >= L.pos) atomicExch(reads_unsolved, 1);
                psrc[idx] = c;
                pval[idx] = val[j0 + i];
            } else {
                psrc[idx] = kPad;
                pval[idx] = VT(0);
            }
        }
        pinv[p] = VT(1) / D[r];
    }
}

// a warp per task: its rows' values and diagonals again
template <typename VT>
__global__ void refill_kernel(const int4 *__restrict__ tasks, int n_tasks, const int *__restrict__ prow,
                              const int *__restrict__ rp, const VT *__restrict__ val, const VT *__restrict__ D,
                              VT *__restrict__ pval, VT *__restrict__ pinv) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int ti = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); ti < n_tasks; ti += nw) {
        const int4 tk = tasks[ti];
        if (lane >= (tk.y & 63)) continue;
        const int p = tk.x + lane, r = prow[p], j0 = rp[r], len = rp[r + 1] - j0 - 1;
        for (int i = 0; i < len; ++i) pval[tk.w + (long long)i * tk.z + lane] = val[j0 + i];
        pinv[p] = VT(1) / D[r];
    }
}

// ------------------------------------------------------------ sync-free --
constexpr int kSfThreads = 256;
constexpr int kSfChunk = 8;   // warp tasks a CTA claims at once (one per warp)
constexpr int kSfEnts = 4;    // entries of a row loaded before its first wait

// "not solved yet": signalling-NaN patterns; arithmetic never returns a
// signalling NaN, so a computed solution is never mistaken for one
template <typename VT> struct Pending;
template <> struct Pending<double> {
    static constexpr unsigned long long bits = 0x7FF5A5A5A5A5A5A5ull;
    __device__ static bool is(double v) { return (unsigned long long)__double_as_longlong(v) == bits; }
    __device__ static double value() { return __longlong_as_double((long long)bits); }
};
template <> struct Pending<float> {
    static constexpr unsigned bits = 0x7FA5A5A5u;
    __device__ static bool is(float v) { return (unsigned)__float_as_uint(v) == bits; }
    __device__ static float value() { return __uint_as_float(bits); }
};

__device__ __forceinline__ double ld_relaxed(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_relaxed(const float *p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_relaxed(double *p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(float *p, float v) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// The value at p once it is no longer pending.  Bounded: after `limit` polls
// the wait records SMAX_ERR_TIMEOUT and raises the abort flag; once the flag
// is up every wait returns NaN (checked every 64 polls).
template <typename VT>
__device__ __noinline__ VT wait_solved(const VT *p, long long limit, int *abort_flag, DevStatus *st) {
    for (long long it = 1;; ++it) {
        if (it > 32) __nanosleep(64);  // the first polls back to back: most waits are short
        const VT v = ld_relaxed(p);
        if (!Pending<VT>::is(v)) return v;
        if ((it & 63) == 0 && *(volatile int *)abort_flag) return VT(NAN);
        if (it >= limit) {
            report(st, SMAX_ERR_TIMEOUT, it);
            atomicExch(abort_flag, 1);
            return VT(NAN);
        }
    }
}

template <typename VT>
__device__ __forceinline__ VT solved(const VT *p, long long limit, int *abort_flag, DevStatus *st) {
    const VT v = ld_relaxed(p);
    return Pending<VT>::is(v) ? wait_solved(p, limit, abort_flag, st) : v;
}

// X := pending; ctl[0] (task counter) = ctl[1] (abort flag) = 0; ctl[4..] pending
template <typename VT>
__global__ void sf_reset_kernel(VT *__restrict__ X, int64_t n, int *__restrict__ ctl) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 == 0) {
        ctl[0] = 0;
        ctl[1] = 0;
        *reinterpret_cast<VT *>(ctl + 4) = Pending<VT>::value();
    }
    for (int64_t i = i0; i < n; i += stride) X[i] = Pending<VT>::value();
}

// ctl: [0] task counter, [1] abort flag, [4..] a word that stays pending
// (waited on by the first row when `never` is set: the test knob).
// A task is (first position, rows | width << 6, level rows = entry stride,
// first entry).
template <typename VT>
__global__ void __launch_bounds__(kSfThreads)
    syncfree_kernel(const int4 *__restrict__ tasks, int n_tasks, const int *__restrict__ prow,
                    const int *__restrict__ psrc, const VT *__restrict__ pval, const VT *__restrict__ pinv,
                    const VT *__restrict__ B, VT *X, int *ctl, long long limit, bool never, DevStatus *st) {
    __shared__ int chunk_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *abort_flag = ctl + 1;
    while (true) {
        if (threadIdx.x == 0) chunk_sh = atomicAdd(ctl, kSfChunk);
        __syncthreads();
        const int c0 = chunk_sh;
        __syncthreads();  // chunk_sh is rewritten on the next turn
        if (c0 >= n_tasks) return;
        const int c1 = min(c0 + kSfChunk, n_tasks);
        for (int ti = c0 + warp; ti < c1; ti += kSfThreads / 32) {
            const int4 tk = tasks[ti];
            const int w = tk.y >> 6;
            if (lane >= (tk.y & 63)) continue;
            // every load goes out before the first wait: entries, then the
            // sources' values, right-hand side and 1/D
            int src[kSfEnts];
            VT v[kSfEnts], xs[kSfEnts];
#pragma unroll
            for (int i = 0; i < kSfEnts; ++i) {
                src[i] = kPad;
                if (i < w) {
                    const long long idx = tk.w + (long long)i * tk.z + lane;
                    src[i] = psrc[idx];
                    v[i] = pval[idx];
                }
            }
#pragma unroll
            for (int i = 0; i < kSfEnts; ++i) xs[i] = src[i] != kPad ? ld_relaxed(X + src[i]) : VT(0);
            const int p = tk.x + lane;
            const int r = prow[p];
            const VT bi = B[r], inv = pinv[p];
            VT sum = VT(0);
            if (never && ti == 0 && lane == 0)
                sum += VT(0) * solved(reinterpret_cast<const VT *>(ctl + 4), limit, abort_flag, st);
            bool more = true;
#pragma unroll
            for (int i = 0; i < kSfEnts; ++i) {
                if (src[i] == kPad) { more = false; break; }
                const VT xv = Pending<VT>::is(xs[i]) ? wait_solved(X + src[i], limit, abort_flag, st) : xs[i];
                sum += v[i] * xv;
            }
            if (more)
                for (int i = kSfEnts; i < w; ++i) {
                    const long long idx = tk.w + (long long)i * tk.z + lane;
                    const int sc = psrc[idx];
                    if (sc == kPad) break;
                    sum += pval[idx] * solved(X + sc, limit, abort_flag, st);
                }
            st_relaxed(X + r, (bi - sum) * inv);
        }
    }
}

// k > 1 right-hand sides, element (r, v) at r*rs + v*vs (row-major: rs = k,
// vs = 1; column-major: rs = 1, vs = the leading dimension): a warp per
// row with its lanes over the vectors, 32 at a time; a CTA claims 8
// consecutive positions, one per warp, with one atomic.  Per row the plain
// solves' arithmetic: x[r][v] = (b[r][v] - sum_j val[j] x[col[j]][v]) / D[r],
// the off-diagonal entries in stored order (the diagonal is last in each row).
template <typename VT>
__global__ void __launch_bounds__(kSfThreads)
    syncfree_rows_kernel(const int *__restrict__ prow, int n, const int *__restrict__ rp, const int *__restrict__ ci,
                         const VT *__restrict__ val, const VT *__restrict__ D, const VT *__restrict__ B, VT *X,
                         int64_t k, int64_t rs, int64_t vs, int *ctl, long long limit, DevStatus *st) {
    __shared__ int base_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *abort_flag = ctl + 1;
    while (true) {
        if (threadIdx.x == 0) base_sh = atomicAdd(ctl, kSfThreads / 32);
        __syncthreads();
        const int p0 = base_sh;
        __syncthreads();  // base_sh is rewritten on the next turn
        if (p0 >= n) return;
        const int p = p0 + warp;
        if (p >= n) continue;
        const int r = prow[p];
        const int s = rp[r], e = rp[r + 1] - 1;
        const VT d = D[r];
        for (int64_t v0 = 0; v0 < k; v0 += 32) {
            const int64_t v = v0 + lane;
            const bool act = v < k;
            VT sum = VT(0);
            for (int j0 = s; j0 < e; j0 += 32) {
                const int jj = j0 + lane;
                const int cj = jj < e ? ci[jj] : 0;
                const VT aj = jj < e ? val[jj] : VT(0);
                const int cnt = min(32, e - j0);
                for (int t = 0; t < cnt; ++t) {
                    const int c = __shfl_sync(0xffffffffu, cj, t);
                    const VT a = __shfl_sync(0xffffffffu, aj, t);
                    if (act) sum += a * solved(X + (int64_t)c * rs + v * vs, limit, abort_flag, st);
                }
            }
            if (act) st_relaxed(X + (int64_t)r * rs + v * vs, (B[(int64_t)r * rs + v * vs] - sum) / d);
        }
    }
}

}  // namespace

bool build_level_pack(LevelPack &pk, const int *rp, const int *ci, const void *val, const void *D, int vbytes,
                      int64_t n, const int *order, const std::vector<int> &src_begin, const std::vector<int> &count,
                      cudaStream_t st) {
    const int L = (int)count.size();
    if ((int)src_begin.size() != L) fail(SMAX_ERR_STATE, "inconsistent sweep steps");
    pk = LevelPack();
    pk.n = n;
    pk.vbytes = vbytes;
    pk.levels = L;
    std::vector<int> pos_begin(L + 1, 0);
    for (int s = 0; s < L; ++s) pos_begin[s + 1] = pos_begin[s] + count[s];
    if (pos_begin[L] != n) fail(SMAX_ERR_STATE, "sweep steps do not cover all rows");
    const size_t nb = sizeof(int) * (n > 0 ? n : 1);
    pk.prow.alloc(nb);
    pk.pinv.alloc((size_t)vbytes * (n > 0 ? n : 1));
    if (n == 0 || L == 0) {
        pk.psrc.alloc(sizeof(int));
        pk.pval.alloc(vbytes);
        return true;
    }
    DevBuf d_pos(sizeof(int) * (L + 1)), d_src(sizeof(int) * L), plev(nb), pos_of_row(nb), len(nb), wmax(sizeof(int) * L);
    SMAX_CUDA(cudaMemcpyAsync(d_pos.p, pos_begin.data(), sizeof(int) * (L + 1), cudaMemcpyHostToDevice, st));
    SMAX_CUDA(cudaMemcpyAsync(d_src.p, src_begin.data(), sizeof(int) * L, cudaMemcpyHostToDevice, st));
    positions_kernel<<<grid_for(n), 256, 0, st>>>(d_pos.as<int>(), L, d_src.as<int>(), order, n, pk.prow.as<int>(),
                                                  plev.as<int>(), pos_of_row.as<int>());
    off_len_kernel<<<grid_for(n), 256, 0, st>>>(rp, pk.prow.as<int>(), n, len.as<int>());
    SMAX_CUDA(cudaGetLastError());
    size_t tb = 0;
    SMAX_CUDA(cub::DeviceSegmentedReduce::Max(nullptr, tb, len.as<int>(), wmax.as<int>(), L, d_pos.as<int>(),
                                              d_pos.as<int>() + 1, st));
    DevBuf tmp(tb);
    SMAX_CUDA(cub::DeviceSegmentedReduce::Max(tmp.p, tb, len.as<int>(), wmax.as<int>(), L, d_pos.as<int>(),
                                              d_pos.as<int>() + 1, st));
    std::vector<int> w(L);
    SMAX_CUDA(cudaMemcpyAsync(w.data(), wmax.p, sizeof(int) * L, cudaMemcpyDeviceToHost, st));
    int h_rp_end = 0;
    SMAX_CUDA(cudaMemcpyAsync(&h_rp_end, rp + n, sizeof(int), cudaMemcpyDeviceToHost, st));
    SMAX_CUDA(cudaStreamSynchronize(st));
    {
        long long padded = 0;
        for (int s = 0; s < L; ++s) padded += (long long)count[s] * (count[s] > 0 ? std::max(w[s], 0) : 0);
        const long long off = (long long)h_rp_end - n;  // off-diagonal entries
        if (padded > 3 * off + (1ll << 20) || padded >= (1ll << 31)) {
            pk = LevelPack();
            return false;
        }
    }
    std::vector<Level> lv(L);
    long long base = 0;
    for (int s = 0; s < L; ++s) {
        const int ws = count[s] > 0 ? std::max(w[s], 0) : 0;
        lv[s] = Level{pos_begin[s], count[s], ws, (int)base};
        base += (long long)count[s] * ws;
    }
    pk.ents = base;
    // warp tasks: (first position, rows | width << 6, entry stride, first entry)
    std::vector<int4> tk;
    tk.reserve((size_t)(n / 32 + L));
    for (int s = 0; s < L; ++s) {
        if (lv[s].w >= (1 << 25)) {  // does not fit the task encoding
            pk = LevelPack();
            return false;
        }
        for (int t0 = 0; t0 < lv[s].m; t0 += 32)
            tk.push_back(make_int4(lv[s].pos + t0, std::min(32, lv[s].m - t0) | (lv[s].w << 6), lv[s].m,
                                   lv[s].base + t0));
    }
    pk.n_tasks = (int)tk.size();
    pk.tasks.alloc(sizeof(int4) * (tk.empty() ? 1 : tk.size()));
    if (!tk.empty())
        SMAX_CUDA(cudaMemcpyAsync(pk.tasks.p, tk.data(), sizeof(int4) * tk.size(), cudaMemcpyHostToDevice, st));
    DevBuf d_lv(sizeof(Level) * L), flag(sizeof(int));
    SMAX_CUDA(cudaMemcpyAsync(d_lv.p, lv.data(), sizeof(Level) * L, cudaMemcpyHostToDevice, st));
    SMAX_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
    pk.psrc.alloc(sizeof(int) * (base > 0 ? base : 1));
    pk.pval.alloc((size_t)vbytes * (base > 0 ? base : 1));
    auto fill = [&](auto zero) {
        using VT = decltype(zero);
        fill_kernel<VT><<<grid_for(n), 256, 0, st>>>(rp, ci, static_cast<const VT *>(val), static_cast<const VT *>(D),
                                                     n, pk.prow.as<int>(), plev.as<int>(), pos_of_row.as<int>(),
                                                     d_lv.as<Level>(), pk.psrc.as<int>(), pk.pval.as<VT>(),
                                                     pk.pinv.as<VT>(), flag.as<int>());
    };
    if (vbytes == 8) fill(0.0);
    else fill(0.0f);
    SMAX_CUDA(cudaGetLastError());
    int h_flag = 0;
    SMAX_CUDA(cudaMemcpyAsync(&h_flag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SMAX_CUDA(cudaStreamSynchronize(st));  // the temporaries die here
    pk.reads_unsolved = h_flag != 0;
    return true;
}

void refill_level_pack(LevelPack &pk, const int *rp, const void *val, const void *D, cudaStream_t st) {
    if (pk.n_tasks == 0) return;
    auto fill = [&](auto zero) {
        using VT = decltype(zero);
        refill_kernel<VT><<<grid_for((int64_t)pk.n_tasks * 32), 256, 0, st>>>(
            pk.tasks.as<int4>(), pk.n_tasks, pk.prow.as<int>(), rp, static_cast<const VT *>(val),
            static_cast<const VT *>(D), pk.pval.as<VT>(), pk.pinv.as<VT>());
    };
    if (pk.vbytes == 8) fill(0.0);
    else fill(0.0f);
    SMAX_CUDA(cudaGetLastError());
}

template <typename VT>
void pack_solve_syncfree(const LevelPack &pk, const VT *B, VT *X, void *ctl, long long limit, bool force_timeout,
                         DevStatus *st, cudaStream_t s) {
    if (pk.n == 0) return;
    int *c = static_cast<int *>(ctl);
    sf_reset_kernel<VT><<<grid_for(pk.n), 256, 0, s>>>(X, pk.n, c);
    static int per_sm_cache[64] = {};
    int dev = 0;
    SMAX_CUDA(cudaGetDevice(&dev));
    int per_sm = dev >= 0 && dev < 64 ? per_sm_cache[dev] : 0;
    if (per_sm == 0) {
        SMAX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, syncfree_kernel<VT>, kSfThreads, 0));
        if (per_sm < 1) per_sm = 1;
        if (dev >= 0 && dev < 64) per_sm_cache[dev] = per_sm;
    }
    const int chunks = (pk.n_tasks + kSfChunk - 1) / kSfChunk;
    // deep, narrow schedules: about four levels' rows in flight, so waiting
    // warps do not flood L2 with polls
    const int64_t avg = pk.n / std::max(1, pk.n_levels());
    const int64_t cap = std::max<int64_t>(8, (4 * avg + kSfThreads - 1) / kSfThreads);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)chunks, (int64_t)per_sm * sm_count(), cap}));
    syncfree_kernel<VT><<<grid, kSfThreads, 0, s>>>(pk.tasks.as<int4>(), pk.n_tasks, pk.prow.as<int>(),
                                                    pk.psrc.as<int>(), pk.pval.as<VT>(), pk.pinv.as<VT>(), B, X, c,
                                                    limit, force_timeout, st);
    SMAX_CUDA(cudaGetLastError());
}

template <typename VT>
void solve_syncfree_rows(const LevelPack &pk, const int *rp, const int *ci, const VT *val, const VT *D, const VT *B,
                         VT *X, int64_t k, bool row_major, void *ctl, long long limit, DevStatus *st, cudaStream_t s) {
    if (pk.n == 0 || k == 0) return;
    int *c = static_cast<int *>(ctl);
    sf_reset_kernel<VT><<<grid_for(pk.n * k), 256, 0, s>>>(X, pk.n * k, c);
    static int per_sm_cache[64] = {};
    int dev = 0;
    SMAX_CUDA(cudaGetDevice(&dev));
    int per_sm = dev >= 0 && dev < 64 ? per_sm_cache[dev] : 0;
    if (per_sm == 0) {
        SMAX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, syncfree_rows_kernel<VT>, kSfThreads, 0));
        if (per_sm < 1) per_sm = 1;
        if (dev >= 0 && dev < 64) per_sm_cache[dev] = per_sm;
    }
    constexpr int rows_per_claim = kSfThreads / 32;
    const int64_t claims = (pk.n + rows_per_claim - 1) / rows_per_claim;
    // about four levels' rows in flight, as for one right-hand side
    const int64_t avg = pk.n / std::max(1, pk.n_levels());
    const int64_t cap = std::max<int64_t>(8, (4 * avg + rows_per_claim - 1) / rows_per_claim);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>({claims, (int64_t)per_sm * sm_count(), cap}));
    // column-major blocks: the leading dimension is the matrix's row count
    const int64_t rs = row_major ? k : 1, vs = row_major ? 1 : pk.n;
    syncfree_rows_kernel<VT><<<grid, kSfThreads, 0, s>>>(pk.prow.as<int>(), (int)pk.n, rp, ci, val, D, B, X, k, rs, vs, c,
                                                         limit, st);
    SMAX_CUDA(cudaGetLastError());
}

template void solve_syncfree_rows<double>(const LevelPack &, const int *, const int *, const double *,
                                          const double *, const double *, double *, int64_t, bool, void *, long long,
                                          DevStatus *, cudaStream_t);
template void solve_syncfree_rows<float>(const LevelPack &, const int *, const int *, const float *, const float *,
                                         const float *, float *, int64_t, bool, void *, long long, DevStatus *,
                                         cudaStream_t);
template void pack_solve_syncfree<double>(const LevelPack &, const double *, double *, void *, long long, bool,
                                          DevStatus *, cudaStream_t);
template void pack_solve_syncfree<float>(const LevelPack &, const float *, float *, void *, long long, bool,
                                         DevStatus *, cudaStream_t);
}  // namespace smax
