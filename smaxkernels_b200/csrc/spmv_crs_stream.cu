// spmv_crs_stream.cu -- CRS SpMV, warp-stream variant (the default on sm_100a).
//
// Reference semantics: SPMV::CPU::naive_crs_spmv
// (src/kernels/spmv/spmv_cpu/spmv_cpu_crs_impl.hpp:9-38): y[i] = sum_j val[j]*x[col[j]].
//
// Design.  The nnz range is cut into fixed slices of W = 512 entries; warp t
// owns slice t, so every warp streams exactly the same number of bytes no
// matter how row lengths are distributed.  A slice is read in chunks of
// 32*U entries, each lane taking U consecutive entries with 128-bit,
// evict-first loads of col and val (the arrays are padded to a multiple of W
// at upload, so the loop has no bounds checks).  Row boundaries come from a
// bit mask built once per matrix: bit e is set when entry e is the last entry
// of its row.  Each lane sums its U products with resets at its row ends; a
// warp-wide segmented scan (shuffles) carries the open partial sum across
// lanes and chunks, and every row that ends inside the slice is written by
// the lane holding its last entry.  The sum a slice holds for the row still
// open at its end is written to carry[t]; a small fix-up pass then adds each
// run of carries to its row in task order (deterministic).  When no row has
// more than 32 entries, a slice instead sums the head of its first row (the
// entries before the slice, at most 31) itself, one entry per lane, and
// neither carries nor the fix-up launch are needed.  Rows without
// entries get y = 0 from a separate list.  Short rows of nearly one length are
// summed by a few lanes each instead (crs_rows_kernel): one launch, no carries,
// no scan.  HBM traffic: val, col, one bit per
// entry, one int per 512 entries, y; x is gathered through L2.
#include "spmv_crs.cuh"

#include <cub/device/device_reduce.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

namespace smax {

namespace {

constexpr int kW = 512;          // entries per warp task
constexpr int kWarpsPerCta = 8;  // 256-thread CTAs

template <typename VT> struct StreamCfg;
template <> struct StreamCfg<double> { static constexpr int U = 4; };
// FP32 lanes take four entries too (16-byte column and value loads): with
// eight, each lane held eight gathers in flight and registers cost occupancy
template <> struct StreamCfg<float> { static constexpr int U = 4; };

// U consecutive entries of col and val starting at a multiple of U.
template <typename VT, int U> struct Chunk;
template <> struct Chunk<double, 4> {
    int c[4];
    double v[4];
    __device__ __forceinline__ void load(const int *col, const double *val, int64_t e) {
        int4 ci = __ldcs(reinterpret_cast<const int4 *>(col + e));
        double2 a = __ldcs(reinterpret_cast<const double2 *>(val + e));
        double2 b = __ldcs(reinterpret_cast<const double2 *>(val + e + 2));
        c[0] = ci.x; c[1] = ci.y; c[2] = ci.z; c[3] = ci.w;
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
};
template <> struct Chunk<float, 4> {
    int c[4];
    float v[4];
    __device__ __forceinline__ void load(const int *col, const float *val, int64_t e) {
        int4 ci = __ldcs(reinterpret_cast<const int4 *>(col + e));
        float4 a = __ldcs(reinterpret_cast<const float4 *>(val + e));
        c[0] = ci.x; c[1] = ci.y; c[2] = ci.z; c[3] = ci.w;
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    }
};

__device__ __forceinline__ int row_of_rank(const int *row_list, int q) { return row_list ? row_list[q] : q; }

// Sum over the entries [rs, base) of the row open at a slice start, one entry
// per lane (base - rs < 32), reduced in a fixed lane order.
template <typename VT>
__device__ __forceinline__ VT head_sum(const int *__restrict__ col, const VT *__restrict__ val,
                                       const VT *__restrict__ x, int64_t rs, int64_t base, int lane) {
    VT h = VT(0);
    if (rs + lane < base) h = __ldg(val + rs + lane) * __ldcg(x + __ldg(col + rs + lane));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    return h;
}

template <typename VT, bool SHORT>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
    crs_stream_kernel(const int *__restrict__ col, const VT *__restrict__ val,
                      const uint32_t *__restrict__ endbits, const int *__restrict__ task_rank,
                      const int *__restrict__ row_list, const int *__restrict__ row_ptr, int64_t n_tasks,
                      int n_nonempty, const VT *__restrict__ x, VT *__restrict__ y, VT *__restrict__ carry_val,
                      int *__restrict__ carry_rank) {
    constexpr int U = StreamCfg<VT>::U;
    constexpr int CH = 32 * U;  // entries per chunk
    constexpr int NC = kW / CH; // chunks per task
    constexpr unsigned MASK = (1u << U) - 1u;
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (t >= n_tasks) return;  // uniform per warp
    const int64_t base = t * kW;
    int q = task_rank[t];      // rank (among non-empty rows) of the row open at the slice start
    VT carry = VT(0);          // partial sum of the open row, from this slice only (SHORT: the whole row)

    Chunk<VT, U> cur;
    int64_t e0 = base + lane * U;
    cur.load(col, val, e0);
    uint32_t word = endbits[e0 >> 5];
    // SHORT: every row has at most 32 entries, so the open row ends in this
    // slice and at most 31 of its entries lie before it
    if constexpr (SHORT) carry = head_sum(col, val, x, (int64_t)row_ptr[row_of_rank(row_list, q)], base, lane);

#pragma unroll
    for (int k = 0; k < NC; ++k) {
        // prefetch the next chunk while this one is reduced
        Chunk<VT, U> nxt;
        uint32_t nword = 0;
        if (k + 1 < NC) {
            nxt.load(col, val, e0 + CH);
            nword = endbits[(e0 + CH) >> 5];
        }
        const unsigned nib = (word >> (unsigned)(e0 & 31)) & MASK;

        VT p[U];
#pragma unroll
        for (int i = 0; i < U; ++i) p[i] = cur.v[i] * __ldcg(x + cur.c[i]);  // L2 only: x lines are not reused in L1

        const int nend = __popc(nib);
        int incl = nend;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int excl = incl - nend;
        const int total_ends = __shfl_sync(0xffffffffu, incl, 31);

        // local segments: head (up to and including the first end), complete
        // rows inside the lane, and the open tail after the last end
        VT run = VT(0), head = VT(0);
        int ri = 0;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            run += p[i];
            if ((nib >> i) & 1u) {
                if (ri == 0) head = run;
                else st_stream(y + row_of_rank(row_list, q + excl + ri), run);
                run = VT(0);
                ++ri;
            }
        }

        // segmented inclusive scan of (v, f) over lanes:
        // (v1,f1) then (v2,f2) -> (f2 ? v2 : v1 + v2, f1 | f2)
        VT sv = run;  // tail if the lane has an end, else its whole sum
        int sf = nend > 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            VT vu = __shfl_up_sync(0xffffffffu, sv, o);
            int fu = __shfl_up_sync(0xffffffffu, sf, o);
            if (lane >= o) {
                if (!sf) sv += vu;
                sf |= fu;
            }
        }
        VT ev = __shfl_up_sync(0xffffffffu, sv, 1);
        int ef = __shfl_up_sync(0xffffffffu, sf, 1);
        if (lane == 0) { ev = VT(0); ef = 0; }
        const VT cin = ef ? ev : carry + ev;
        if (nend) st_stream(y + row_of_rank(row_list, q + excl), cin + head);

        const VT v31 = __shfl_sync(0xffffffffu, sv, 31);
        const int f31 = __shfl_sync(0xffffffffu, sf, 31);
        carry = f31 ? v31 : carry + v31;
        q += total_ends;

        if (k + 1 < NC) {
            cur = nxt;
            word = nword;
            e0 += CH;
        }
    }
    if (!SHORT && lane == 0) {
        carry_val[t] = carry;
        carry_rank[t] = q < n_nonempty ? q : -1;
    }
}

// Short rows (at most 32 entries) of nearly one length, G lanes a row: lane l
// takes the row's entries l, l + G, ..., at most U of them (G * U >= the longest
// row), all loaded before any is used.  The lanes of a warp read neighbouring
// rows, so every line of col and val is used up from L1, and the x entries that
// neighbouring rows of a grid share are found there too.  Bound by HBM: 190^3
// 7-point FP64 171 -> 136 us (5.2 TB/s of val, col, row_ptr, x and y).
template <typename VT, int G, int U>
__global__ void __launch_bounds__(256) crs_rows_kernel(const int *__restrict__ col, const VT *__restrict__ val,
                                                       const int *__restrict__ row_ptr, int64_t n,
                                                       const VT *__restrict__ x, VT *__restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t row = i / G;
    const int gl = (int)(i % G);
    int s = 0, e = 0;
    if (row < n) {
        s = row_ptr[row] + gl;
        e = row_ptr[row + 1];
    }
    int c[U];
    VT v[U], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (s + u * G < e) {
            c[u] = __ldg(col + s + u * G);
            v[u] = __ldg(val + s + u * G);
        }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (s + u * G < e) xv[u] = __ldg(x + c[u]);
    VT sum = VT(0);
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (s + u * G < e) sum += v[u] * xv[u];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (row < n && gl == 0) st_stream(y + row, sum);
}

// y[row] += the run of carries of one row, summed in task order.
template <typename VT>
__global__ void crs_stream_fixup(const VT *__restrict__ carry_val, const int *__restrict__ carry_rank,
                                 const int *__restrict__ row_list, int64_t n_tasks, VT *__restrict__ y) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tasks) return;
    const int q = carry_rank[t];
    if (q < 0 || (t > 0 && carry_rank[t - 1] == q)) return;
    VT s = VT(0);
    for (int64_t u = t; u < n_tasks && carry_rank[u] == q; ++u) s += carry_val[u];
    y[row_of_rank(row_list, q)] += s;
}

template <typename VT>
__global__ void zero_rows(const int *__restrict__ rows, int64_t n, VT *__restrict__ y) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[rows[i]] = VT(0);
}

__global__ void row_flags_kernel(const int *__restrict__ row_ptr, int64_t n, unsigned char *__restrict__ empty,
                                 unsigned char *__restrict__ nonempty, uint32_t *__restrict__ endbits,
                                 int *__restrict__ max_len) {
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int len = 0;
    if (r < n) {
        const int s = row_ptr[r], e = row_ptr[r + 1];
        const bool em = e == s;
        empty[r] = em;
        nonempty[r] = !em;
        if (!em) atomicOr(endbits + ((e - 1) >> 5), 1u << ((e - 1) & 31));
        len = e - s;
    }
    len = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);
    if ((threadIdx.x & 31) == 0 && len > 0) atomicMax(max_len, len);
}

// A sample of the columns, 32 neighbouring rows a warp: found[0] counts entries of
// rows short enough for crs_rows_kernel, found[1] those whose column lies more
// than kFar from that of the row before's entry in the same place, found[2] rows,
// found[3] those whose columns span at most narrow_width an entry.
constexpr int kFar = 16384;
// The columns an entry up to which a matrix of rows of len entries is better streamed
// (crs_spmv_stream).  Of a multiple of four entries, a stream's lanes, of four each,
// gather neighbouring rows' neighbouring columns together; rows that leave a third of
// crs_rows_kernel's slots unused cost it more.  Others gather worse than it does, unless
// their columns follow on each other (12 million entries FP64, stream and rows: of 27,
// 37 apart, 59 and 43, neighbours 38 and 41).
__device__ __forceinline__ int narrow_width(int len) {
    if (len == 8 || len == 16) return 80;
    const int slots = len <= 4 ? 4 : (len <= 8 ? 8 : (len <= 16 ? 16 : 32));
    return len % 4 == 0 || 3 * len < 2 * slots ? 40 : 4;
}
constexpr int kSampleWarps = 512;
__global__ void scatter_sample_kernel(const int *__restrict__ row_ptr, const int *__restrict__ col, int64_t n,
                                      int *__restrict__ found) {
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t r = (n > 32 ? (n - 32) * w / kSampleWarps : 0) + lane;
    int s = 0, len = 0;
    if (r < n) {
        s = row_ptr[r];
        len = min(row_ptr[r + 1] - s, 32);
    }
    int seen = 0, far = 0, lo = INT_MAX, hi = -1;
    const int most = __reduce_max_sync(0xffffffffu, len);
    for (int i = 0; i < most; ++i) {
        const int c = i < len ? col[s + i] : -1;
        if (c >= 0) {
            lo = min(lo, c);
            hi = max(hi, c);
        }
        const int before = __shfl_up_sync(0xffffffffu, c, 1);
        if (lane > 0 && c >= 0 && before >= 0) {
            ++seen;
            far += abs(c - before) > kFar;
        }
    }
    seen = __reduce_add_sync(0xffffffffu, seen);
    far = __reduce_add_sync(0xffffffffu, far);
    const int rows = __popc(__ballot_sync(0xffffffffu, hi >= 0));
    const int close = __popc(__ballot_sync(0xffffffffu, hi >= 0 && hi - lo <= narrow_width(len) * len));
    if (lane == 0) {
        atomicAdd(found, seen);
        atomicAdd(found + 1, far);
        atomicAdd(found + 2, rows);
        atomicAdd(found + 3, close);
    }
}

// rank of the row holding entry t*W: the largest r with row_ptr[r] <= t*W
// (that row is non-empty), then its position among the non-empty rows.
__global__ void task_rank_kernel(const int *__restrict__ row_ptr, int64_t n, const int *__restrict__ row_list,
                                 int64_t n_nonempty, int64_t n_tasks, int *__restrict__ task_rank) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tasks) return;
    const int64_t e = t * kW;
    int64_t lo = 0, hi = n;  // upper_bound over row_ptr[0..n]
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if ((int64_t)row_ptr[mid] <= e) lo = mid + 1; else hi = mid;
    }
    int64_t r = lo - 1;
    if (row_list) {
        int64_t a = 0, b = n_nonempty;  // lower_bound of r in row_list
        while (a < b) {
            int64_t m = (a + b) >> 1;
            if (row_list[m] < r) a = m + 1; else b = m;
        }
        r = a;
    }
    task_rank[t] = (int)r;
}

}  // namespace

int crs_stream_pad() { return kW; }

void CrsStreamPlan::build(const int *d_row_ptr, int64_t n, int64_t nnz_, int vbytes, cudaStream_t st,
                          const int *d_col) {
    n_rows = n;
    nnz = nnz_;
    n_tasks = (nnz + kW - 1) / kW;
    int64_t words = (n_tasks * kW) / 32 + 1;
    endbits.alloc(sizeof(uint32_t) * words);
    SMAX_CUDA(cudaMemsetAsync(endbits.p, 0, endbits.bytes, st));
    n_empty = 0;
    n_nonempty = 0;
    row_ptr = d_row_ptr;
    longest = 0;
    scattered = narrow = false;
    if (n > 0) {
        DevBuf fe(n), fne(n), cnt(sizeof(int) * 7);
        SMAX_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes, st));
        row_flags_kernel<<<ceil_div_u(n, 256), 256, 0, st>>>(d_row_ptr, n, fe.as<unsigned char>(),
                                                             fne.as<unsigned char>(), endbits.as<uint32_t>(),
                                                             cnt.as<int>() + 2);
        if (d_col)
            scatter_sample_kernel<<<kSampleWarps / 8, 256, 0, st>>>(d_row_ptr, d_col, n, cnt.as<int>() + 3);
        SMAX_CUDA(cudaGetLastError());
        thrust::counting_iterator<int> it(0);
        empty_rows.alloc(sizeof(int) * n);
        size_t tb = 0;
        SMAX_CUDA(cub::DeviceSelect::Flagged(nullptr, tb, it, fe.as<unsigned char>(), empty_rows.as<int>(),
                                             cnt.as<int>(), (int)n, st));
        DevBuf tmp(tb);
        SMAX_CUDA(cub::DeviceSelect::Flagged(tmp.p, tb, it, fe.as<unsigned char>(), empty_rows.as<int>(),
                                             cnt.as<int>(), (int)n, st));
        int h[7] = {0, 0, 0, 0, 0, 0, 0};
        SMAX_CUDA(cudaMemcpyAsync(h, cnt.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        SMAX_CUDA(cudaStreamSynchronize(st));
        n_empty = h[0];
        longest = h[2];
        scattered = 2 * h[4] > h[3];
        narrow = 2 * h[6] > h[5];
        n_nonempty = n - n_empty;
        if (n_empty > 0) {
            row_list.alloc(sizeof(int) * (n_nonempty > 0 ? n_nonempty : 1));
            SMAX_CUDA(cub::DeviceSelect::Flagged(tmp.p, tb, it, fne.as<unsigned char>(), row_list.as<int>(),
                                                 cnt.as<int>() + 1, (int)n, st));
        } else {
            empty_rows.release();
            row_list.release();
        }
        SMAX_CUDA(cudaStreamSynchronize(st));
    }
    task_rank.alloc(sizeof(int) * (n_tasks > 0 ? n_tasks : 1));
    carry_rank.alloc(sizeof(int) * (n_tasks > 0 ? n_tasks : 1));
    carry_val.alloc((size_t)vbytes * (n_tasks > 0 ? n_tasks : 1));
    if (n_tasks > 0) {
        task_rank_kernel<<<ceil_div_u(n_tasks, 256), 256, 0, st>>>(
            d_row_ptr, n, row_list.p ? row_list.as<int>() : nullptr, n_nonempty, n_tasks, task_rank.as<int>());
        SMAX_CUDA(cudaGetLastError());
    }
    SMAX_CUDA(cudaStreamSynchronize(st));
}

template <typename VT>
void crs_spmv_stream(const CrsStreamPlan &p, const int *col, const VT *val, const VT *x, VT *y, cudaStream_t st) {
    // Rows of nearly one length, up to 32: a lane (or 2, 4) per row.  Lanes left
    // without entries cost as much as the others, so only where rows are two
    // thirds full on average.  B200, us, stream -> rows: 128^3 7-point FP64
    // (98% full) 54.8 -> 48.1, 96^3 27-point 86.3 -> 70.9, 2^20 rows of 5, one in
    // 100 of 7 (72%) 32.3 -> 25.0; 2^22 rows of 0 to 32 evenly (50%) 299 -> 318,
    // of 2, one in 100 of 32 (7%) 57 -> 229.  Columns all over a large x push a row's
    // own lines out of L1 before its lanes have used them: 2^20 rows of 17 FP64 88 ->
    // 107, of 32 150 -> 172 (of 8 45 -> 47, and 2^17 rows of 32 30 -> 30).
    const bool crowded = p.scattered && p.longest > 8 && p.n_rows >= (1 << 18);
    // Columns close together are in L1 either way, and the stream loads col and val
    // better.  Rows of 8, 16 and, in FP32, 32 entries put a warp's loads on few of L1's
    // banks (columns 37 apart, 4 million entries FP64: of 8 21 and 24, of 16 21 and 24;
    // below a million 12 and 12); beyond L2 other lengths lose as well (12 million FP64: of
    // 9 42 and 51, of 12 41 and 45; FP32: of 2 31 and 48, of 12 28 and 30; 4 million
    // FP64: of 12 22 and 18).
    const bool banks = p.longest == 8 || p.longest == 16 || (p.longest == 32 && sizeof(VT) == 4);
    const bool beyond = p.nnz * (int64_t)(sizeof(VT) + sizeof(int)) >= (int64_t)80 << 20;
    const bool streams = p.narrow && (beyond || (banks && p.nnz >= (1 << 20)));
    if (p.n_rows > 0 && p.longest <= 32 && !crowded && !streams && 3 * p.nnz >= 2 * p.n_rows * p.longest) {
        // rows without entries get their zero here as well
        auto rows = [&](auto kern, int g) {
            kern<<<ceil_div_u((uint64_t)p.n_rows * g, 256), 256, 0, st>>>(col, val, p.row_ptr, p.n_rows, x, y);
            SMAX_CUDA(cudaGetLastError());
        };
        if (p.longest <= 4) rows(crs_rows_kernel<VT, 1, 4>, 1);
        else if (p.longest <= 8) rows(crs_rows_kernel<VT, 1, 8>, 1);
        else if (p.longest <= 16) rows(crs_rows_kernel<VT, 2, 8>, 2);
        else rows(crs_rows_kernel<VT, 4, 8>, 4);
        return;
    }
    const int *rl = p.row_list.p ? p.row_list.as<int>() : nullptr;
    if (p.n_tasks > 0) {
        unsigned grid = ceil_div_u(p.n_tasks, kWarpsPerCta);
        auto launch = [&](auto kern) {
            kern<<<grid, kWarpsPerCta * 32, 0, st>>>(col, val, p.endbits.as<uint32_t>(), p.task_rank.as<int>(), rl,
                                                     p.row_ptr, p.n_tasks, (int)p.n_nonempty, x, y,
                                                     p.carry_val.as<VT>(), p.carry_rank.as<int>());
            SMAX_CUDA(cudaGetLastError());
        };
        if (p.longest <= 32) {
            launch(crs_stream_kernel<VT, true>);  // no carries: one launch
        } else {
            launch(crs_stream_kernel<VT, false>);
            crs_stream_fixup<VT><<<ceil_div_u(p.n_tasks, 256), 256, 0, st>>>(
                p.carry_val.as<VT>(), p.carry_rank.as<int>(), rl, p.n_tasks, y);
            SMAX_CUDA(cudaGetLastError());
        }
    }
    if (p.n_empty > 0) {
        zero_rows<VT><<<ceil_div_u(p.n_empty, 256), 256, 0, st>>>(p.empty_rows.as<int>(), p.n_empty, y);
        SMAX_CUDA(cudaGetLastError());
    }
}

template void crs_spmv_stream<double>(const CrsStreamPlan &, const int *, const double *, const double *, double *,
                                      cudaStream_t);
template void crs_spmv_stream<float>(const CrsStreamPlan &, const int *, const float *, const float *, float *,
                                     cudaStream_t);

}  // namespace smax
