// spmv_bcrs.cu -- BCRS SpMV and CRS -> BCRS conversion on sm_100a.
//
// Layout (src/common.hpp:90-111, src/utils/convert_formats.hpp:134-247): block
// row r holds blocks row_ptr[r]..row_ptr[r+1]-1; block j is the hpad x wpad
// tile val[j*hpad*wpad ...] stored row-major (ix*wpad+jx) or column-major
// (jx*hpad+ix); x is indexed by col[j]*wpad+jx and y by r*hpad+ix, for
// ix < bh and jx < bw (SPMV::CPU::naive_bcrs_spmv,
// src/kernels/spmv/spmv_cpu/spmv_cpu_bcrs_impl.hpp:19-85).
//
// SpMV, register-blocked block-row stream (block size bs = hpad*wpad divisible
// by VEC = 16/sizeof(VT) and dividing 32*VEC, e.g. 4x4): one warp per block
// row streams that row's blocks as one flat array with 128-bit evict-first
// loads; because the warp advances 32*VEC values per step, every lane always
// sees the same VEC in-block positions, so it keeps VEC register accumulators
// for fixed (ix, jx).  Lanes holding the same positions combine with
// shuffles; the bs partial sums are then folded into the bh outputs through
// a per-warp shared-memory tile (fixed order, deterministic).  Long block
// rows (three or more warp steps on average) use a four-step loop with more
// loads in flight; short ones (under two steps: e.g. a stencil in 4x4 blocks)
// give each block row a group of bs/VEC lanes instead of a warp.  Other block
// sizes up to kMaxBs give a lane each in-block position; larger ones, and many
// short block rows, one thread per block row in the reference's loop order.
//
// Conversion: per block row, the sorted distinct block columns of its bh rows
// (segmented radix sort of col/bw over the block row's entries, then a
// uniqueness pass and a scan), then every entry is written into its block at
// the in-block index of the chosen order; blocks are zero-filled first.
#include "spmv_formats.cuh"

#include <algorithm>
#include <type_traits>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_radix_sort.cuh>
#include <cub/device/device_select.cuh>

namespace smax {

namespace {

template <typename VT> struct V16;
template <> struct V16<double> { using T = double2; static constexpr int N = 2; };
template <> struct V16<float> { using T = float4; static constexpr int N = 4; };

// Block values: evict-first (streamed once), or with KEEP the default
// policy, so that a matrix whose values fit in L2 stays there across products.
template <typename VT, int VEC, bool KEEP = false>
__device__ __forceinline__ void load16(const VT *p, VT *o) {
    if constexpr (VEC == 2) {
        const double2 *q = reinterpret_cast<const double2 *>(p);
        const double2 v = KEEP ? __ldg(q) : __ldcs(q);
        o[0] = v.x; o[1] = v.y;
    } else {
        const float4 *q = reinterpret_cast<const float4 *>(p);
        const float4 v = KEEP ? __ldg(q) : __ldcs(q);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
}

constexpr int kMaxBs = 128;  // largest block size of the stream and lane paths

// How a lane reads the x values of its VEC consecutive in-block positions.
enum XMode {
    kEach = 0,  // one load per position that is inside the block (padded blocks, odd shapes)
    kRow = 1,   // row-major unpadded: VEC consecutive x values, one 16-byte load
    kCol = 2,   // column-major unpadded: all VEC positions lie in one column, one value
};

template <typename VT, int XM> struct XVals {
    static constexpr int VEC = V16<VT>::N;
    VT v[XM == kCol ? 1 : VEC];
    __device__ __forceinline__ void load(const VT *xb, const int (&jx)[VEC], const bool (&ok)[VEC]) {
        if constexpr (XM == kRow) {
            load16<VT, VEC, true>(xb + jx[0], v);
        } else if constexpr (XM == kCol) {
            v[0] = ld_keep(xb + jx[0]);
        } else {
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[i] = ok[i] ? ld_keep(xb + jx[i]) : VT(0);
        }
    }
    __device__ __forceinline__ void add(const VT (&a)[VEC], const bool (&ok)[VEC], VT (&acc)[VEC]) const {
#pragma unroll
        for (int i = 0; i < VEC; ++i)
            if (XM != kEach || ok[i]) acc[i] += a[i] * v[XM == kCol ? 0 : i];
    }
};

// The rows a warp takes: order[w], order[w + W], ... of a grid of W warps
// (longest first, so the long rows start first and the strided shares are
// even).  A row's bounds are loaded while the row before it is summed.
struct RowWalk {
    const int *__restrict__ row_ptr;
    const int *__restrict__ order;
    int64_t n, w, W;
    int row, b0, b1;  // the current row
    int nrow, nb0, nb1;
    __device__ __forceinline__ void fetch() {
        nrow = -1;
        nb0 = nb1 = 0;
        if (w < n) {
            nrow = order ? order[w] : (int)w;
            nb0 = row_ptr[nrow];
            nb1 = row_ptr[nrow + 1];
        }
        w += W;
    }
    __device__ __forceinline__ void next() {
        row = nrow;
        b0 = nb0;
        b1 = nb1;
        fetch();
    }
    __device__ RowWalk(const int *rp, const int *ord, int64_t n_rows) : row_ptr(rp), order(ord), n(n_rows) {
        w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        W = (int64_t)gridDim.x * (blockDim.x >> 5);
        fetch();
        next();
    }
};

// The stream loop, a warp per block row.  bs is a power of two here, so a
// warp step covers a whole number of blocks and a lane's block advances by a
// constant: no index division in the loop.  U steps' values and x entries are
// loaded before any is used (the last steps of a row are masked, not looped
// over one by one), and the column indices one iteration ahead -- the next
// row's first ones during this row's last iteration -- so the x gathers wait
// on no load of their own.  Bound by HBM and, between rows, by latency; four
// steps on three CTAs an SM fill it (five CTAs spill: 168 us in the first
// line).  B200, before (a warp per row, one step's indexes and gathers at a
// time) and now, us: 27-point grid 48^3 in 4x4 blocks FP64 114 -> 78, FP32
// 157 -> 54; 28^3 in 8x8 FP64 65 -> 55; 2^22 rows of lognormal length in 4x4
// FP64 2080 -> 1557.
template <typename VT, int XM, bool KEEP, int U, int CTAS>
__global__ void __launch_bounds__(256, CTAS) bcrs_stream_kernel(const int *__restrict__ row_ptr,
                                                                const int *__restrict__ col,
                                                                const VT *__restrict__ val, int64_t n_brows, int bh,
                                                                int bw, int hpad, int wpad, int col_major,
                                                                const VT *__restrict__ x, VT *__restrict__ y,
                                                                const int *__restrict__ order) {
    constexpr int VEC = V16<VT>::N;
    __shared__ VT tile[8][kMaxBs];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int bs = hpad * wpad;
    const int o = (lane * VEC) & (bs - 1);  // this lane's first in-block position
    int jx[VEC];
    bool ok[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int q = o + i;
        const int ix = col_major ? q % hpad : q / wpad;
        jx[i] = col_major ? q / hpad : q % wpad;
        ok[i] = ix < bh && jx[i] < bw;
    }
    const int per = 32 * VEC / bs;    // blocks of a warp step
    const int sub = lane * VEC / bs;  // this lane's block of a step
    const int groups = bs / VEC;      // lanes l and l + groups*m hold the same positions
    RowWalk rows(row_ptr, order, n_brows);
    int cn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int j = rows.b0 + sub + u * per;
        cn[u] = j < rows.b1 ? col[j] : 0;
    }
    while (rows.row >= 0) {  // uniform per warp
        const int br = rows.row, b1 = rows.b1;
        VT acc[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] = VT(0);
        int j0 = rows.b0;
        const VT *vp = val + (int64_t)(j0 + sub) * bs + o;
        do {
            const int j = j0 + sub;
            VT v[U][VEC];
            XVals<VT, XM> xv[U];
            const VT *xb[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u * per < b1) {
                    load16<VT, VEC, KEEP>(vp + u * 32 * VEC, v[u]);
                    xb[u] = x + (int64_t)cn[u] * wpad;
                }
            j0 += U * per;
            const bool more = j0 < b1;
            // the columns after these: of this row, or the first of the next
            const int jn = (more ? j0 : rows.nb0) + sub, bn = more ? b1 : rows.nb1;
#pragma unroll
            for (int u = 0; u < U; ++u) cn[u] = jn + u * per < bn ? col[jn + u * per] : 0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u * per < b1) xv[u].load(xb[u], jx, ok);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u * per < b1) xv[u].add(v[u], ok, acc);
            vp += U * 32 * VEC;
        } while (j0 < b1);
        rows.next();
        for (int s = groups; s < 32; s <<= 1)
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], s);
        if (lane < groups)
#pragma unroll
            for (int i = 0; i < VEC; ++i) tile[warp][o + i] = acc[i];
        __syncwarp();
        for (int ix = lane; ix < bh; ix += 32) {
            VT s = VT(0);
            for (int q = 0; q < bw; ++q) s += tile[warp][col_major ? q * hpad + ix : ix * wpad + q];
            st_stream(y + (int64_t)br * hpad + ix, s);
        }
        __syncwarp();  // the tile is written again for the next row
    }
}

// Other block sizes up to kMaxBs, a lane per in-block position, so that the
// loads of a step are contiguous.  NS == 1, blocks of at most 32 values: G
// lanes per block row, G / bs blocks a step, 32 / G block rows a warp: the
// whole warp, or for short block rows bs lanes each (several rows side by
// side).  NS > 1: a block a step, NS positions a lane.  U steps' loads are in
// flight, and the column indices come one iteration ahead.  3x3 blocks, before
// (a thread per block row, its values strided) and now, us: 27-point grid 48^3
// FP64 169 -> 91, FP32 125 -> 79; 7-point 64^3 FP64 84 -> 63.
template <typename VT, int NS, int U>
__global__ void __launch_bounds__(256) bcrs_lane_kernel(const int *__restrict__ row_ptr, const int *__restrict__ col,
                                                        const VT *__restrict__ val, int64_t n_brows, int bh, int bw,
                                                        int hpad, int wpad, int col_major, const VT *__restrict__ x,
                                                        VT *__restrict__ y, const int *__restrict__ order, int G) {
    __shared__ VT tile[8][NS * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int bs = hpad * wpad;
    const int rows = 32 / G, g = lane / G, gl = lane - g * G;
    const int64_t w = ((int64_t)blockIdx.x * 8 + warp) * rows + g;
    const bool has = g < rows && w < n_brows;
    const int64_t br = has ? (order ? order[w] : w) : 0;
    const int per = NS == 1 ? G / bs : 1;  // blocks of a step
    const int sub = NS == 1 ? gl / bs : 0;
    int jx[NS];
    bool ok[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        const int q = NS == 1 ? gl - sub * bs : lane + 32 * i;
        const int ix = col_major ? q % hpad : q / wpad;
        jx[i] = col_major ? q / hpad : q % wpad;
        ok[i] = has && sub < per && q < bs && ix < bh && jx[i] < bw;
    }
    VT acc[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) acc[i] = VT(0);
    int j0 = has ? row_ptr[br] : 0;
    const int b1 = has ? row_ptr[br + 1] : 0;
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = j0 + u * per + sub < b1 ? col[j0 + u * per + sub] : -1;
    for (; j0 < b1; j0 += U * per) {
        VT v[U][NS], xv[U][NS];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const VT *p = val + (int64_t)(j0 + u * per) * bs + gl;
#pragma unroll
            for (int i = 0; i < NS; ++i)
                if (ok[i] && c[u] >= 0) {
                    v[u][i] = ld_stream(p + 32 * i);
                    xv[u][i] = ld_keep(x + (int64_t)c[u] * wpad + jx[i]);
                }
        }
        int cn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + (U + u) * per + sub;
            cn[u] = j < b1 ? col[j] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int i = 0; i < NS; ++i)
                if (ok[i] && c[u] >= 0) acc[i] += v[u][i] * xv[u][i];
            c[u] = cn[u];
        }
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) tile[warp][lane + 32 * i] = acc[i];
    __syncwarp();
    if (has)
        for (int ix = gl; ix < bh; ix += G) {
            VT s = VT(0);
            for (int q = 0; q < bw; ++q)
                for (int b = 0; b < per; ++b)
                    s += tile[warp][g * G + b * bs + (col_major ? q * hpad + ix : ix * wpad + q)];
            st_stream(y + br * hpad + ix, s);
        }
}

// Short block rows: a group of G = bs / VEC lanes per block row (8 lanes for
// 4x4 FP64), one block per step, two blocks' loads in flight.  Every lane
// keeps the same VEC in-block positions for the whole row, so the bs sums
// are complete without shuffles and are folded into the bh outputs through
// the group's shared-memory tile (fixed order).
template <typename VT, bool KEEP>
__global__ void __launch_bounds__(256) bcrs_group_kernel(const int *__restrict__ row_ptr,
                                                         const int *__restrict__ col, const VT *__restrict__ val,
                                                         int64_t n_brows, int bh, int bw, int hpad, int wpad,
                                                         int col_major, const VT *__restrict__ x,
                                                         VT *__restrict__ y) {
    constexpr int VEC = V16<VT>::N;
    __shared__ VT tile[256 * VEC];  // 256 / G groups x bs values = 256 * VEC
    const int bs = hpad * wpad;
    const int G = bs / VEC;
    const int g_in_cta = threadIdx.x / G, lg = threadIdx.x % G;
    const int64_t br = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int o = lg * VEC;
    int jx[VEC];
    bool ok[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int q = o + i;
        const int ix = col_major ? q % hpad : q / wpad;
        jx[i] = col_major ? q / hpad : q % wpad;
        ok[i] = ix < bh && jx[i] < bw;
    }
    VT acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = VT(0);
    if (br < n_brows) {
        const int b1 = row_ptr[br + 1];
        int j = row_ptr[br];
        for (; j + 1 < b1; j += 2) {
            VT v0[VEC], v1[VEC];
            load16<VT, VEC, KEEP>(val + (int64_t)j * bs + o, v0);
            load16<VT, VEC, KEEP>(val + (int64_t)(j + 1) * bs + o, v1);
            const int64_t c0 = (int64_t)col[j] * wpad, c1 = (int64_t)col[j + 1] * wpad;
            VT x0[VEC], x1[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                x0[i] = ok[i] ? ld_keep(x + c0 + jx[i]) : VT(0);
                x1[i] = ok[i] ? ld_keep(x + c1 + jx[i]) : VT(0);
            }
#pragma unroll
            for (int i = 0; i < VEC; ++i)
                if (ok[i]) {
                    acc[i] += v0[i] * x0[i];
                    acc[i] += v1[i] * x1[i];
                }
        }
        if (j < b1) {
            VT v[VEC];
            load16<VT, VEC, KEEP>(val + (int64_t)j * bs + o, v);
            const int64_t c = (int64_t)col[j] * wpad;
#pragma unroll
            for (int i = 0; i < VEC; ++i)
                if (ok[i]) acc[i] += v[i] * ld_keep(x + c + jx[i]);
        }
    }
    VT *t = tile + g_in_cta * bs;
#pragma unroll
    for (int i = 0; i < VEC; ++i) t[o + i] = acc[i];
    __syncthreads();
    if (br < n_brows)
        for (int ix = lg; ix < bh; ix += G) {
            VT s = VT(0);
            for (int q = 0; q < bw; ++q) s += t[col_major ? q * hpad + ix : ix * wpad + q];
            st_stream(y + br * hpad + ix, s);
        }
}

// block sizes beyond kMaxBs, and many short block rows: one thread per block
// row, the reference's loop order
template <typename VT>
__global__ void bcrs_thread_kernel(const int *__restrict__ row_ptr, const int *__restrict__ col,
                                   const VT *__restrict__ val, int64_t n_brows, int bh, int bw, int hpad, int wpad,
                                   int col_major, const VT *__restrict__ x, VT *__restrict__ y) {
    const int64_t br = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (br >= n_brows) return;
    const int64_t bs = (int64_t)hpad * wpad;
    for (int ix = 0; ix < bh; ++ix) {
        VT s = VT(0);
        for (int j = row_ptr[br]; j < row_ptr[br + 1]; ++j) {
            const VT *blk = val + (int64_t)j * bs;
            const VT *xb = x + (int64_t)col[j] * wpad;
            for (int jx = 0; jx < bw; ++jx) s += blk[col_major ? jx * hpad + ix : ix * wpad + jx] * xb[jx];
        }
        y[br * hpad + ix] = s;
    }
}

// ----------------------------------------------------------- conversion ----
__global__ void bcrs_keys(const int *__restrict__ row_ptr, const int *__restrict__ col, int64_t n, int bw,
                          int *__restrict__ keys) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    for (int j = row_ptr[r] + lane; j < row_ptr[r + 1]; j += 32) keys[j] = col[j] / bw;
}

__global__ void bcrs_seg_offsets(const int *__restrict__ row_ptr, int64_t n_brows, int bh, int *__restrict__ off) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b <= n_brows) off[b] = row_ptr[b * bh];
}

// flag[j] = 1 when sorted[j] starts a new distinct block column in its block row
__global__ void bcrs_unique_flags(const int *__restrict__ sorted, const int *__restrict__ off, int64_t n_brows,
                                  int64_t nnz, unsigned char *__restrict__ flag, int *__restrict__ brow_of) {
    const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (b >= n_brows) return;
    for (int64_t j = off[b] + lane; j < off[b + 1]; j += 32) {
        flag[j] = (j == off[b] || sorted[j] != sorted[j - 1]) ? 1 : 0;
        brow_of[j] = (int)b;
    }
}

__global__ void bcrs_count(const int *__restrict__ brow_of_unique, int64_t n_unique, int *__restrict__ counts) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u < n_unique) atomicAdd(counts + brow_of_unique[u], 1);
}

__global__ void bcrs_ptr(const int *__restrict__ incl, int64_t n_brows, int *__restrict__ b_row_ptr) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b <= n_brows) b_row_ptr[b] = b == 0 ? 0 : incl[b - 1];
}

template <typename VT>
__global__ void bcrs_fill(const int *__restrict__ row_ptr, const int *__restrict__ col, const VT *__restrict__ val,
                          int64_t n, int bh, int bw, int hpad, int wpad, int col_major,
                          const int *__restrict__ b_row_ptr, const int *__restrict__ b_col, VT *__restrict__ b_val) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const int64_t br = r / bh;
    const int lr = (int)(r % bh);
    const int64_t bs = (int64_t)hpad * wpad;
    for (int j = row_ptr[r] + lane; j < row_ptr[r + 1]; j += 32) {
        const int bc = col[j] / bw;
        int lo = b_row_ptr[br], hi = b_row_ptr[br + 1];
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (b_col[mid] < bc) lo = mid + 1; else hi = mid;
        }
        const int in = col_major ? hpad * (col[j] % bw) + lr : wpad * lr + col[j] % bw;
        b_val[(int64_t)lo * bs + in] = val[j];
    }
}

}  // namespace

bool bcrs_stream_path(int64_t hpad, int64_t wpad, int vbytes) {
    const int vec = 16 / vbytes;
    const int64_t bs = hpad * wpad;
    return bs > 0 && bs <= kMaxBs && bs % vec == 0 && (32 * vec) % bs == 0;
}

template <typename VT>
void bcrs_spmv(const DevBCRS &m, const VT *x, VT *y, cudaStream_t st) {
    if (m.n_rows == 0) return;
    const int *order = m.order.p ? m.order.as<int>() : nullptr;
    const int64_t bs = m.hpad * m.wpad;
    constexpr int VEC = 16 / (int)sizeof(VT);
    // a warp per block row, longest rows first; as many CTAs as are resident
    auto go = [&](auto kern, int per_sm) {
        const uint64_t grid = std::min<uint64_t>(((uint64_t)m.n_rows + 7) / 8, (uint64_t)per_sm * sm_count());
        kern<<<(unsigned)grid, 256, 0, st>>>(m.row_ptr.as<int>(), m.col.as<int>(), m.val.as<VT>(), m.n_rows,
                                             (int)m.bh, (int)m.bw, (int)m.hpad, (int)m.wpad, m.col_major ? 1 : 0, x, y,
                                             order);
    };
    // A thread or a lane per position (block sizes off the stream path): a thread's
    // time grows with a row's values, which its warp reads strided and must find in
    // L1 again; that of the lanes with the number of rows, a warp each above 16 values
    // a block, of which every chunk of rows pays its latency.  Blocks of up to 16
    // values, thread / lanes, us: 3x3, one a row, 20000 rows FP32 10 / 12, 80000 12 / 20; five a
    // row, 20000 16 / 14, 80000 22 / 24; FP64 of 2^19 rows, four a row 100 / 92, seven 194 / 117.
    // Larger ones: 5x5, one a row, 8000 rows FP32 12 / 14, 20000 12 / 18; three a row, 8000
    // 17 / 14, 20000 18 / 19, 40000 22 / 28, 2^19 129 / 247, FP64 216 / 272, and four 307 / 281;
    // five, FP32 247 / 292; 7x7, 2.3 a row, 40000 rows FP32 30 / 26, 80000 40 / 43, 2^19 FP64
    // 298 / 293, three a row 397 / 344, FP32 304 / 270.
    const bool int_end = near_int_end(m.n_blocks);
    const int64_t most_vals = bs <= 16 ? std::min<int64_t>(256 / (int64_t)sizeof(VT), m.n_rows / 1500)
                                       : std::min<int64_t>(sizeof(VT) == 4 ? 128 : 112, m.n_rows / 400);
    const bool thread_rows = int_end || (m.n_blocks * bs <= most_vals * m.n_rows &&
                                         (bs <= 16 || sizeof(VT) == 4 || m.n_blocks < 4 * m.n_rows));
    // a lane per in-block position, `lanes` lanes per block row
    auto go_lanes = [&](auto kern, int lanes) {
        kern<<<ceil_div_u(m.n_rows, 8 * (32 / lanes)), 256, 0, st>>>(
            m.row_ptr.as<int>(), m.col.as<int>(), m.val.as<VT>(), m.n_rows, (int)m.bh, (int)m.bw, (int)m.hpad,
            (int)m.wpad, m.col_major ? 1 : 0, x, y, order, lanes);
    };
    if (bcrs_stream_path(m.hpad, m.wpad, sizeof(VT)) && !int_end) {
        // mean warp steps per block row: below two a lane group per block row
        // wastes fewer lanes; more loads in flight pay off from about three
        const double steps = (double)m.n_blocks * (double)bs / ((double)m.n_rows * 32.0 * VEC);
        // values that fit in half of L2 are loaded with the default policy and
        // stay resident across repeated products (4x4 blocks of the 7-point
        // 64^3 Laplacian, 59 MB of values, in a loop of products: see the
        // BCRS notes); larger ones stream evict-first
        const bool keep = (double)m.n_blocks * (double)bs * sizeof(VT) <= 0.5 * (double)l2_bytes();
        const bool whole = m.bh == m.hpad && m.bw == m.wpad;
        const int xm = !whole ? kEach
                       : m.col_major ? (m.hpad % VEC == 0 ? kCol : kEach)
                       : (m.wpad % VEC == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) ? kRow : kEach;
        auto with_x = [&](auto f) {
            if (xm == kRow) f(std::integral_constant<int, kRow>());
            else if (xm == kCol) f(std::integral_constant<int, kCol>());
            else f(std::integral_constant<int, kEach>());
        };
        if (steps < 2.0) {
            const uint64_t threads = (uint64_t)m.n_rows * (uint64_t)(bs / VEC);
            auto kern = keep ? bcrs_group_kernel<VT, true> : bcrs_group_kernel<VT, false>;
            kern<<<ceil_div_u(threads, 256), 256, 0, st>>>(m.row_ptr.as<int>(), m.col.as<int>(), m.val.as<VT>(),
                                                           m.n_rows, (int)m.bh, (int)m.bw, (int)m.hpad, (int)m.wpad,
                                                           m.col_major ? 1 : 0, x, y);
        } else {
            with_x([&](auto XM) {
                if (steps < 3.0 && keep) go(bcrs_stream_kernel<VT, XM.value, true, 2, 4>, 4);
                else if (steps < 3.0) go(bcrs_stream_kernel<VT, XM.value, false, 2, 4>, 4);
                else if (keep) go(bcrs_stream_kernel<VT, XM.value, true, 4, 3>, 3);
                else go(bcrs_stream_kernel<VT, XM.value, false, 4, 3>, 3);
            });
        }
    } else if (bs <= 32 && !thread_rows) {
        // several block rows a warp: fewer than three warp steps a block row, or more
        // where there are rows for all warps (2^19 rows of nine 3x3 blocks FP64: 135 us,
        // 260 with a warp each; 27 of them on 160000 rows 88 and 131; 1000 rows 13.6 and 11.7)
        const int64_t per = 32 / bs;
        const bool many = bs <= 16 && m.n_rows >= 64ll * sm_count() && m.n_blocks <= 32 * m.n_rows;
        go_lanes(bcrs_lane_kernel<VT, 1, 4>, many || m.n_blocks < 3 * per * m.n_rows ? (int)bs : 32);
    } else if (bs <= 64 && !thread_rows) {
        go_lanes(bcrs_lane_kernel<VT, 2, 2>, 32);
    } else if (bs <= kMaxBs && !thread_rows) {
        go_lanes(bcrs_lane_kernel<VT, 4, 1>, 32);
    } else {
        bcrs_thread_kernel<VT><<<ceil_div_u(m.n_rows, 128), 128, 0, st>>>(
            m.row_ptr.as<int>(), m.col.as<int>(), m.val.as<VT>(), m.n_rows, (int)m.bh, (int)m.bw, (int)m.hpad,
            (int)m.wpad, m.col_major ? 1 : 0, x, y);
    }
    SMAX_CUDA(cudaGetLastError());
}

namespace {
__global__ void bcrs_row_lengths(const int *__restrict__ row_ptr, int64_t n, int *__restrict__ len,
                                 int *__restrict__ idx) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    len[r] = row_ptr[r + 1] - row_ptr[r];
    idx[r] = (int)r;
}
}  // namespace

void bcrs_plan(DevBCRS &m, cudaStream_t st) {
    m.order.release();
    if (m.n_rows < 2) return;
    const int64_t n = m.n_rows;
    DevBuf len(sizeof(int) * n), idx(sizeof(int) * n), len_sorted(sizeof(int) * n);
    m.order.alloc(sizeof(int) * n);
    bcrs_row_lengths<<<ceil_div_u(n, 256), 256, 0, st>>>(m.row_ptr.as<int>(), n, len.as<int>(), idx.as<int>());
    SMAX_CUDA(cudaGetLastError());
    size_t tb = 0;
    SMAX_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, len.as<int>(), len_sorted.as<int>(),
                                                        idx.as<int>(), m.order.as<int>(), (int)n, 0, 32, st));
    DevBuf tmp(tb ? tb : 1);
    SMAX_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.p, tb, len.as<int>(), len_sorted.as<int>(),
                                                        idx.as<int>(), m.order.as<int>(), (int)n, 0, 32, st));
    SMAX_CUDA(cudaStreamSynchronize(st));
}

template void bcrs_spmv<double>(const DevBCRS &, const double *, double *, cudaStream_t);
template void bcrs_spmv<float>(const DevBCRS &, const float *, float *, cudaStream_t);

void crs_to_bcrs(const DevCRS &a, int vbytes, int64_t bh, int64_t bw, int64_t hpad, int64_t wpad, bool col_major,
                 DevBCRS &out, cudaStream_t st, int64_t max_blocks) {
    // the reference throws for these (src/utils/convert_formats.hpp:143-160); it
    // tests the height padding twice, this platform tests both paddings
    if (bh <= 0 || bw <= 0 || a.n_rows % bh) fail(SMAX_ERR_BAD_ARG, "Target block height does not divide number of input rows");
    if (a.n_cols % bw) fail(SMAX_ERR_BAD_ARG, "Target block width does not divide number of input columns");
    if (hpad < bh) fail(SMAX_ERR_BAD_ARG, "Height padding has to be at least target block height");
    if (wpad < bw) fail(SMAX_ERR_BAD_ARG, "Width padding has to be at least target block width");
    const int64_t n = a.n_rows, nnz = a.nnz, nb = n / bh;
    out.n_rows = nb;
    out.n_cols = a.n_cols / bw;
    out.bh = bh; out.bw = bw; out.hpad = hpad; out.wpad = wpad;
    out.col_major = col_major;
    out.row_ptr.alloc(sizeof(int) * (nb + 1));
    if (nnz == 0) {
        SMAX_CUDA(cudaMemsetAsync(out.row_ptr.p, 0, sizeof(int) * (nb + 1), st));
        out.n_blocks = 0;
        SMAX_CUDA(cudaStreamSynchronize(st));
        return;
    }
    DevBuf keys(sizeof(int) * nnz), sorted(sizeof(int) * nnz), off(sizeof(int) * (nb + 1));
    bcrs_keys<<<ceil_div_u((uint64_t)n * 32, 256), 256, 0, st>>>(a.rp(), a.ci(), n, (int)bw, keys.as<int>());
    bcrs_seg_offsets<<<ceil_div_u(nb + 1, 256), 256, 0, st>>>(a.rp(), nb, (int)bh, off.as<int>());
    SMAX_CUDA(cudaGetLastError());
    size_t tb = 0;
    SMAX_CUDA(cub::DeviceSegmentedRadixSort::SortKeys(nullptr, tb, keys.as<int>(), sorted.as<int>(), (int)nnz,
                                                      (int)nb, off.as<int>(), off.as<int>() + 1, 0, 32, st));
    DevBuf tmp(tb);
    SMAX_CUDA(cub::DeviceSegmentedRadixSort::SortKeys(tmp.p, tb, keys.as<int>(), sorted.as<int>(), (int)nnz,
                                                      (int)nb, off.as<int>(), off.as<int>() + 1, 0, 32, st));
    DevBuf flag(nnz), brow(sizeof(int) * nnz), ucol(sizeof(int) * nnz), ubrow(sizeof(int) * nnz), nsel(sizeof(int) * 2);
    bcrs_unique_flags<<<ceil_div_u((uint64_t)nb * 32, 256), 256, 0, st>>>(sorted.as<int>(), off.as<int>(), nb, nnz,
                                                                          flag.as<unsigned char>(), brow.as<int>());
    SMAX_CUDA(cudaGetLastError());
    size_t tb2 = 0;
    SMAX_CUDA(cub::DeviceSelect::Flagged(nullptr, tb2, sorted.as<int>(), flag.as<unsigned char>(), ucol.as<int>(),
                                         nsel.as<int>(), (int)nnz, st));
    DevBuf tmp2(tb2);
    SMAX_CUDA(cub::DeviceSelect::Flagged(tmp2.p, tb2, sorted.as<int>(), flag.as<unsigned char>(), ucol.as<int>(),
                                         nsel.as<int>(), (int)nnz, st));
    SMAX_CUDA(cub::DeviceSelect::Flagged(tmp2.p, tb2, brow.as<int>(), flag.as<unsigned char>(), ubrow.as<int>(),
                                         nsel.as<int>() + 1, (int)nnz, st));
    int nu = 0;
    SMAX_CUDA(cudaMemcpyAsync(&nu, nsel.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SMAX_CUDA(cudaStreamSynchronize(st));
    out.n_blocks = nu;
    if (max_blocks >= 0 && nu > max_blocks) {
        // more blocks than the caller accepts: report the count, build nothing
        out.col.release();
        out.val.release();
        return;
    }
    DevBuf counts(sizeof(int) * nb), incl(sizeof(int) * nb);
    SMAX_CUDA(cudaMemsetAsync(counts.p, 0, sizeof(int) * nb, st));
    bcrs_count<<<ceil_div_u(nu, 256), 256, 0, st>>>(ubrow.as<int>(), nu, counts.as<int>());
    SMAX_CUDA(cudaGetLastError());
    size_t tb3 = 0;
    SMAX_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tb3, counts.as<int>(), incl.as<int>(), (int)nb, st));
    DevBuf tmp3(tb3);
    SMAX_CUDA(cub::DeviceScan::InclusiveSum(tmp3.p, tb3, counts.as<int>(), incl.as<int>(), (int)nb, st));
    bcrs_ptr<<<ceil_div_u(nb + 1, 256), 256, 0, st>>>(incl.as<int>(), nb, out.row_ptr.as<int>());
    SMAX_CUDA(cudaGetLastError());
    out.col.alloc(sizeof(int) * nu);
    SMAX_CUDA(cudaMemcpyAsync(out.col.p, ucol.p, sizeof(int) * nu, cudaMemcpyDeviceToDevice, st));
    const int64_t bs = hpad * wpad;
    out.val.alloc((size_t)vbytes * nu * bs);
    SMAX_CUDA(cudaMemsetAsync(out.val.p, 0, (size_t)vbytes * nu * bs, st));
    const unsigned grid = ceil_div_u((uint64_t)n * 32, 256);
    if (vbytes == 8)
        bcrs_fill<double><<<grid, 256, 0, st>>>(a.rp(), a.ci(), a.val.as<double>(), n, (int)bh, (int)bw, (int)hpad,
                                                (int)wpad, col_major, out.row_ptr.as<int>(), out.col.as<int>(),
                                                out.val.as<double>());
    else
        bcrs_fill<float><<<grid, 256, 0, st>>>(a.rp(), a.ci(), a.val.as<float>(), n, (int)bh, (int)bw, (int)hpad,
                                               (int)wpad, col_major, out.row_ptr.as<int>(), out.col.as<int>(),
                                               out.val.as<float>());
    SMAX_CUDA(cudaGetLastError());
    SMAX_CUDA(cudaStreamSynchronize(st));
}

}  // namespace smax

namespace smax {
namespace {
__global__ void validate_bcrs_kernel(const int *__restrict__ rp, const int *__restrict__ col, int64_t n,
                                     int64_t n_blocks, int64_t n_cols, DevStatus *st) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0 && (rp[0] != 0 || rp[n] != n_blocks)) report(st, SMAX_ERR_BAD_ARG, 0);
    for (int64_t r = t; r < n; r += stride)
        if (rp[r + 1] < rp[r]) report(st, SMAX_ERR_BAD_ARG, r);
    for (int64_t j = t; j < n_blocks; j += stride) {
        const int c = col[j];
        if (c < 0 || c >= n_cols) report(st, SMAX_ERR_COL_OOB, j);
    }
}
}  // namespace

void validate_bcrs(const DevBCRS &m, DevStatus *st, cudaStream_t s) {
    validate_bcrs_kernel<<<4 * sm_count(), 256, 0, s>>>(m.row_ptr.as<int>(), m.col.as<int>(), m.n_rows, m.n_blocks,
                                                        m.n_cols, st);
    SMAX_CUDA(cudaGetLastError());
}
}  // namespace smax
