// sweep.cu -- level-ordered packed triangular solves on sm_100a.
//
// The per-row recurrence is the reference's (naive_crs_sptrsv / crs_sptrsv_lvl,
// src/kernels/sptrsv/sptrsv_cpu/sptrsv_cpu_crs_impl.hpp:9-55,
// sptrsv_lvl_cpu_crs_impl.hpp:11-82): x[r] = (b[r] - sum_j val[j] x[col[j]]) / D[r]
// with the off-diagonal entries summed in stored order.  What changes is the
// layout, for latency: thousands of narrow levels are a chain of dependent
// steps, so a run of them is swept by one CTA, and a level should cost only
// what its successor has to wait for:
//
//   * solutions a row needs are read from the shared-memory ring of the last
//     kRing positions (a slot is safe while q >= level_end - kRing; in a level of
//     more than kRing positions, whose chunks are stored in no order, only its
//     first kRing have a slot that no other of the level writes);
//   * every other operand is in shared memory already: some warps issue bulk
//     copies (cp.async.bulk, completion on an mbarrier) of whole records, as
//     far ahead as the stage has room, and needs no register of the others;
//   * the solving warps form kGroups groups that take the chunks of rows in
//     turn.  A group reads its next chunk's header and operands into registers
//     while other groups solve the chunks before it; then it waits for the
//     level before its own (an mbarrier per level), and between that and the
//     arrival the next level waits for lie only the ring reads, the sum and
//     the store.
//
// Several right-hand sides are independent sweeps: one CTA each, reading the
// same pack through L2.
//
// What bounds it: narrow levels by the chain wait, ring read, sum, store,
// arrive, 0.22 us a level; wide ones by the SM's issue slots (62% busy at up to
// 1024 rows a level) and L1 (67%).  B200, 5-point D+L
// in natural order, FP64; before: one CTA whose threads load every level from
// global memory two levels ahead and meet at a barrier.
//     100^2 (199 levels)             124 -> 48 us
//     512^2                          727 -> 226 us
//     2048^2 (4095 levels)          5020 -> 2400 us
//     1024^2, 32 right-hand sides   2900 -> 1490 us
//     48 matrices in one batch       919 -> 370 us
#include "sweep.cuh"

#include <algorithm>

#include <cub/device/device_segmented_reduce.cuh>

#include "tma.cuh"

namespace smax {

namespace {

constexpr int kRing = SweepPack::kRing;
constexpr int kHeader = 48;   // bytes of a chunk's header
constexpr int kSlots = 32;    // mbarriers of records
constexpr int kWindow = 14;   // records in flight: the first not given back and those after it
constexpr int kLevels = 4;    // levels in flight (mbarriers): one is solved, the next is waited for
constexpr int kGroups = SweepPack::kGroups;
constexpr int kCopyWarps = 4;  // 2048^2 natural, records of 1/16 of the stage: 5.59 ms with 1, 3.96 with 2, 3.37 with 4
// a group polls the level before its chunk's at most kGroups levels past the
// last one known to be solved: no earlier phase of that mbarrier is open
static_assert(kLevels >= kGroups && kSlots >= kWindow + kGroups, "mbarriers for the groups' lead");
// A copying warp before record i may still have to see that record
// i - kCopyWarps - kWindow + 1 was given back, while the others have issued up
// to i + kWindow - 1: the mbarrier must not have been used again by then.
static_assert(kSlots > 2 * kWindow + kCopyWarps - 2, "mbarriers for the copying warps' lead");
constexpr int kRecChunks = 32;             // chunks of a record, at most
// Time of a level, in steps of 10 ns, up to which it is swept: a quarter of
// the waits' default limit, since the threads of a run wait while one of them
// goes through a row of a million entries.
constexpr long long kLevelTime = 1 << 26;
// Arrivals of a phase that an mbarrier counts, one of them the test's that never comes.
constexpr int kMaxArrivals = (1 << 20) - 2;
// An arrived copy takes microseconds; a CTA does not end before its own have.
constexpr long long kDrainNs = 2000000000ll;

// header flags (the width is above them)
constexpr int kFlagBits = 4;
enum : int {
    kRingOnly = 1,  // no entry reads x from global memory
    kDirect = 2,    // too wide for the stage: read in place
    kTwo = 4,       // layout of at most two entries a row
    kThree = 8,     // layout of three
};

struct ChunkDesc {  // what the fill kernels and the header need
    int pos, m, w, mp;
    int off;                // blob offset / 16
    int lpos, lend, rpos;   // positions of the level, first position of the run
    int flags, next, boff, level;  // next, boff: stage offsets of the group's next chunk, of the right-hand sides
    int next_rec;           // the next chunk's record in the run
    int rec_arrive, lev_arrive, pad;  // arrivals each warp owes the record and the level
};
static_assert(sizeof(ChunkDesc) == 64, "four 16-byte loads");

// bytes of a chunk's data per (padded) row
__host__ __device__ constexpr int row_bytes(int flags, int w, int vb) {
    return flags & kTwo ? (vb == 8 ? 32 : 20) : (flags & kThree ? (vb == 8 ? 48 : 32) : w * (vb + 4) + vb);
}

struct Record {
    int off, bytes, pos, bbytes;  // blob offset / 16, bytes, first position, bytes of right-hand sides
    int stage, dep, from, pad;    // stage offset; records [from, dep) of the run must be given back first (all before `from` were)
};
static_assert(sizeof(Record) == 32, "two 16-byte loads");

unsigned grid_for(int64_t work) {
    const int64_t cap = (int64_t)sm_count() * 8;
    const int64_t g = (work + 255) / 256;
    return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

// ---------------------------------------------------------------- build ----
// row, and position of each row, for every position of every chunk
__global__ void sw_positions_kernel(const ChunkDesc *__restrict__ ch, const int *__restrict__ chunk_src,
                                    const int *__restrict__ pchunk, const int *__restrict__ order, int64_t npos,
                                    int *__restrict__ prow, int *__restrict__ pos_of_row) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += stride) {
        const int c = pchunk[p];
        const int t = (int)p - ch[c].pos;
        int r = -1;
        if (t < ch[c].m) {
            const int k = chunk_src[c] + t;
            r = order ? order[k] : k;
            pos_of_row[r] = (int)p;
        }
        prow[p] = r;
    }
}

__global__ void sw_off_len_kernel(const int *__restrict__ rp, const int *__restrict__ order, int64_t n,
                                  int *__restrict__ len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int r = order ? order[k] : (int)k;
        len[k] = rp[r + 1] - rp[r] - 1;
    }
}

// Where entry i's value and source code and the diagonal of row t lie.
//   kTwo    FP64: {v0 v1}[mp] {d s0 s1}[mp]         FP32: {v0 v1 s0 s1}[mp] d[mp]
//   kThree  FP64: {v0 v1}[mp] {v2 d}[mp] {s0 s1 s2 -}[mp]   FP32: {v0 v1 v2 d}[mp] {s0 s1 s2 -}[mp]
//   else    v[w][mp] d[mp] s[w][mp]
// The first two are 16-byte elements, one load each.
template <typename VT> struct RowSlots {
    unsigned char *data;
    int flags, w, mp, t;
    static constexpr int VB = sizeof(VT);
    __device__ VT *value(int i) const {
        if (flags & (kTwo | kThree)) {
            const int per = 16 / VB;  // values of an element
            return reinterpret_cast<VT *>(data + ((int64_t)(i / per) * mp + t) * 16) + i % per;
        }
        return reinterpret_cast<VT *>(data) + (int64_t)i * mp + t;
    }
    __device__ VT *diag() const {
        if (flags & kTwo)
            return VB == 8 ? reinterpret_cast<VT *>(data + ((int64_t)mp + t) * 16)
                           : reinterpret_cast<VT *>(data + (int64_t)mp * 16) + t;
        if (flags & kThree) return value(3);
        return reinterpret_cast<VT *>(data) + (int64_t)w * mp + t;
    }
    __device__ int *source(int i) const {
        if (flags & kTwo)
            return reinterpret_cast<int *>(data + ((int64_t)(VB == 8 ? mp : 0) + t) * 16) + 2 + i;
        if (flags & kThree)
            return reinterpret_cast<int *>(data + ((int64_t)(VB == 8 ? 2 : 1) * mp + t) * 16) + i;
        return reinterpret_cast<int *>(data + (int64_t)(w + 1) * mp * VB) + (int64_t)i * mp + t;
    }
};

// One position's entries.  PATTERN: source codes too (and which chunks read
// global solutions); otherwise new values only.  wraps: some level of a run has
// more than kRing positions.
template <typename VT, bool PATTERN>
__global__ void sw_fill_kernel(const int *__restrict__ rp, const int *__restrict__ ci, const VT *__restrict__ val,
                               const VT *__restrict__ D, int64_t npos, const int *__restrict__ prow,
                               const int *__restrict__ pchunk, const int *__restrict__ pos_of_row,
                               const ChunkDesc *__restrict__ ch, unsigned char *__restrict__ blob, bool div,
                               bool wraps, int *__restrict__ reads_global, int *__restrict__ needs_init) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += stride) {
        const int r = prow[p];
        if (r < 0) continue;
        const ChunkDesc c = ch[pchunk[p]];
        const RowSlots<VT> to{blob + (int64_t)c.off * 16 + kHeader, c.flags, c.w, c.mp, (int)p - c.pos};
        const int j0 = rp[r], len = rp[r + 1] - j0 - 1;
        const int width = c.flags & kTwo ? 2 : c.w;
        for (int i = 0; i < width; ++i) {
            *to.value(i) = i < len ? val[j0 + i] : VT(0);
            if (PATTERN) {
                int code = kRing * (int)sizeof(VT);
                if (i < len) {
                    const int q = pos_of_row[ci[j0 + i]];
                    if (q >= c.lpos) atomicExch(needs_init, 1);
                    bool ring = q >= c.rpos && q < c.lpos && q >= c.lend - kRing;
                    if (ring && wraps) ring = q - ch[pchunk[q]].lpos < kRing;
                    code = ring ? (q & (kRing - 1)) * (int)sizeof(VT) : ~q;
                    if (!ring) reads_global[pchunk[p]] = 1;
                }
                *to.source(i) = code;
            }
        }
        *to.diag() = div ? D[r] : VT(1) / D[r];
    }
}

__global__ void sw_header_kernel(const ChunkDesc *__restrict__ ch, int n_chunks, const int *__restrict__ reads_global,
                                 unsigned char *__restrict__ blob) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_chunks) return;
    const ChunkDesc d = ch[c];
    const int flags = d.flags | (reads_global[c] ? 0 : kRingOnly);
    int4 *h = reinterpret_cast<int4 *>(blob + (int64_t)d.off * 16);
    h[0] = make_int4(d.pos, d.m, (d.w << kFlagBits) | flags, d.next);
    h[1] = make_int4(d.boff, d.level, d.next_rec, d.rec_arrive);
    h[2] = make_int4(d.lev_arrive, d.off, 0, 0);
}

// ------------------------------------------------- gather and scatter ------
// one right-hand side
template <typename VT>
__global__ void sw_gather1_kernel(const int *__restrict__ prow, int64_t npos, const VT *__restrict__ B,
                                  VT *__restrict__ bp, const VT *__restrict__ X, VT *__restrict__ xp) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += stride) {
        const int r = prow[p];
        bp[p] = r >= 0 ? B[r] : VT(0);
        if (xp) xp[p] = r >= 0 ? X[r] : VT(0);
    }
}

template <typename VT>
__global__ void sw_scatter1_kernel(const int *__restrict__ prow, int64_t npos, const VT *__restrict__ xp,
                                   VT *__restrict__ X) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += stride) {
        const int r = prow[p];
        if (r >= 0) X[r] = xp[p];
    }
}

// several: 32 positions by 32 right-hand sides through shared memory, both sides coalesced
template <typename VT>
__global__ void __launch_bounds__(256) sw_gather_kernel(const int *__restrict__ prow, int64_t npos,
                                                        const VT *__restrict__ B, VT *__restrict__ bp,
                                                        const VT *__restrict__ X, VT *__restrict__ xp, int64_t k,
                                                        int64_t rs, int64_t vs) {
    __shared__ VT tb[32][33], tx[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t tiles = (npos + 31) / 32;
    const int64_t v0 = (int64_t)blockIdx.y * 32;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t p0 = tile * 32;
        for (int i = w; i < 32; i += 8) {
            // row-major blocks: lanes over vectors; column-major: lanes over positions
            const int64_t p = p0 + (vs == 1 ? i : lane), v = v0 + (vs == 1 ? lane : i);
            const int r = p < npos ? prow[p] : -1;
            const bool ok = r >= 0 && v < k;
            tb[p - p0][v - v0] = ok ? B[r * rs + v * vs] : VT(0);
            if (xp) tx[p - p0][v - v0] = ok ? X[r * rs + v * vs] : VT(0);
        }
        __syncthreads();
        for (int i = w; i < 32; i += 8) {
            const int64_t p = p0 + lane, v = v0 + i;
            if (p < npos && v < k) {
                bp[v * npos + p] = tb[lane][i];
                if (xp) xp[v * npos + p] = tx[lane][i];
            }
        }
        __syncthreads();
    }
}

template <typename VT>
__global__ void __launch_bounds__(256) sw_scatter_kernel(const int *__restrict__ prow, int64_t npos,
                                                         const VT *__restrict__ xp, VT *__restrict__ X, int64_t k,
                                                         int64_t rs, int64_t vs) {
    __shared__ VT tx[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t tiles = (npos + 31) / 32;
    const int64_t v0 = (int64_t)blockIdx.y * 32;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t p0 = tile * 32;
        for (int i = w; i < 32; i += 8) {
            const int64_t p = p0 + lane, v = v0 + i;
            if (p < npos && v < k) tx[lane][i] = xp[v * npos + p];
        }
        __syncthreads();
        for (int i = w; i < 32; i += 8) {
            const int64_t p = p0 + (vs == 1 ? i : lane), v = v0 + (vs == 1 ? lane : i);
            const int r = p < npos ? prow[p] : -1;
            if (r >= 0 && v < k) X[r * rs + v * vs] = tx[p - p0][v - v0];
        }
        __syncthreads();
    }
}

template <typename VT>
void sw_gather(const SweepPack &pk, const VT *B, const VT *X, int64_t k, int64_t rs, int64_t vs, cudaStream_t st) {
    const int *prow = pk.prow.as<int>();
    VT *bp = pk.bp.as<VT>(), *xp = pk.needs_x_init ? pk.xp.as<VT>() : nullptr;
    if (k == 1 && rs == 1)
        sw_gather1_kernel<VT><<<grid_for(pk.npos), 256, 0, st>>>(prow, pk.npos, B, bp, X, xp);
    else
        sw_gather_kernel<VT><<<dim3(grid_for(pk.npos * 8), (unsigned)((k + 31) / 32)), 256, 0, st>>>(prow, pk.npos, B,
                                                                                                    bp, X, xp, k, rs, vs);
}

template <typename VT>
void sw_scatter(const SweepPack &pk, VT *X, int64_t k, int64_t rs, int64_t vs, cudaStream_t st) {
    const int *prow = pk.prow.as<int>();
    const VT *xp = pk.xp.as<VT>();
    if (k == 1 && rs == 1)
        sw_scatter1_kernel<VT><<<grid_for(pk.npos), 256, 0, st>>>(prow, pk.npos, xp, X);
    else
        sw_scatter_kernel<VT><<<dim3(grid_for(pk.npos * 8), (unsigned)((k + 31) / 32)), 256, 0, st>>>(prow, pk.npos, xp,
                                                                                                     X, k, rs, vs);
}

template <typename VT, bool DIV> __device__ __forceinline__ VT finish_row(VT b, VT sum, VT d) {
    return DIV ? (b - sum) / d : (b - sum) * d;
}

// ---------------------------------------------------------- wide levels ----
constexpr int kWideEnts = 4;  // entries of a row whose loads are all issued before the first use

// one wide level: thread per row.  The first kWideEnts entries and their
// solutions are loaded before any is used, so a row costs one entry load and
// one gather of latency instead of one pair per entry.
template <typename VT, bool DIV>
__global__ void __launch_bounds__(256, 8) sw_wide_kernel(SweepPack::Wide L, const unsigned char *__restrict__ blob, int64_t npos,
                               const VT *__restrict__ bp, VT *xp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.m) return;
    const unsigned char *data = blob + (int64_t)L.off * 16 + kHeader;
    const VT *pv = reinterpret_cast<const VT *>(data) + t;
    const int *ps = reinterpret_cast<const int *>(data + (int64_t)(L.w + 1) * L.mp * (int)sizeof(VT)) + t;
    const int64_t p = blockIdx.y * npos + L.pos + t;
    VT *x = xp + blockIdx.y * npos;
    int src[kWideEnts];
    VT v[kWideEnts], xs[kWideEnts];
#pragma unroll
    for (int i = 0; i < kWideEnts; ++i) {
        src[i] = 0;  // codes of a wide level name positions (negative) or padding
        if (i < L.w) {
            src[i] = ps[i * L.mp];  // (a pack has less than 2^31 entries)
            v[i] = pv[i * L.mp];
        }
    }
#pragma unroll
    for (int i = 0; i < kWideEnts; ++i) xs[i] = src[i] < 0 ? x[~src[i]] : VT(0);
    const VT b = bp[p], d = pv[L.w * L.mp];
    VT sum = VT(0);
    bool more = true;
#pragma unroll
    for (int i = 0; i < kWideEnts; ++i) {
        if (src[i] >= 0) { more = false; break; }
        sum += v[i] * xs[i];
    }
    if (more)
        for (int i = kWideEnts; i < L.w; ++i) {
            const int s = ps[i * L.mp];
            if (s >= 0) break;
            sum += pv[i * L.mp] * x[~s];
        }
    xp[p] = finish_row<VT, DIV>(b, sum, d);
}

// The same of longer rows: kLongEnts entries and their solutions at a time, the
// next entries on their way while these are added.  64 threads a CTA, so that a
// level of a few hundred rows still spreads over the SMs.  Bound by the latency of
// the gathers: 600 rows of 40 random sources FP64 5.3 us a level, of 200 24 us.
constexpr int kLongEnts = 16;
template <typename VT, bool DIV>
__global__ void __launch_bounds__(64) sw_wide_long_kernel(SweepPack::Wide L, const unsigned char *__restrict__ blob,
                                                          int64_t npos, const VT *__restrict__ bp, VT *xp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.m) return;
    const unsigned char *data = blob + (int64_t)L.off * 16 + kHeader;
    const VT *pv = reinterpret_cast<const VT *>(data) + t;
    const int *ps = reinterpret_cast<const int *>(data + (int64_t)(L.w + 1) * L.mp * (int)sizeof(VT)) + t;
    const int64_t p = blockIdx.y * npos + L.pos + t;
    VT *x = xp + blockIdx.y * npos;
    const VT b = bp[p], d = pv[(int64_t)L.w * L.mp];
    int src[kLongEnts];
    VT v[kLongEnts], sum = VT(0);
    auto fetch = [&](int i0) {
#pragma unroll
        for (int i = 0; i < kLongEnts; ++i) {
            src[i] = 0;  // padding
            v[i] = VT(0);
            if (i0 + i < L.w) {
                src[i] = ps[(int64_t)(i0 + i) * L.mp];
                v[i] = pv[(int64_t)(i0 + i) * L.mp];
            }
        }
    };
    fetch(0);
    for (int i0 = 0; i0 < L.w; i0 += kLongEnts) {
        VT xs[kLongEnts], w[kLongEnts];
#pragma unroll
        for (int i = 0; i < kLongEnts; ++i) {
            xs[i] = src[i] < 0 ? x[~src[i]] : VT(0);
            w[i] = v[i];
        }
        const bool last = src[kLongEnts - 1] >= 0;  // the row ends here
        if (!last) fetch(i0 + kLongEnts);
#pragma unroll
        for (int i = 0; i < kLongEnts; ++i) sum += w[i] * xs[i];
        if (last) break;
    }
    xp[p] = finish_row<VT, DIV>(b, sum, d);
}

// ----------------------------------------------------------------- runs ----
// Shared state of a sweeping CTA, at the start of its dynamic shared memory.
struct SweepShared {
    unsigned long long full[kSlots];   // a record has arrived
    unsigned long long empty[kSlots];  // its operands are no longer needed
    unsigned long long level[kLevels]; // a level is solved
    long long wait_ns;  // a wait gives up after this time
    int failed;  // a wait gave up
    int mat, rec0, level0;  // batch: the matrix taken, records and levels before it
};
constexpr int kSharedBytes = 640;
static_assert(sizeof(SweepShared) <= kSharedBytes, "shared state");

template <typename VT> constexpr int ring_bytes() { return (kRing + 16 / (int)sizeof(VT)) * (int)sizeof(VT); }

__device__ __forceinline__ void bulk_copy(unsigned dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ uint64_t *as_bar(unsigned long long *p) { return reinterpret_cast<uint64_t *>(p); }

__device__ __forceinline__ long long sw_now() {
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

constexpr int kPolls = 16;  // polls of a wait between two looks at the time
constexpr unsigned kWarp = 0xffffffffu;

__device__ __forceinline__ int sw_failed(const SweepShared *sh) { return *(const volatile int *)&sh->failed; }

// Whether a wait that began at t0 (0: begins now) is over without what it waits
// for: its time is up or another thread's was.  Returns when it began, 0 when it
// is over.
__device__ __noinline__ long long sw_patience(SweepShared *sh, long long t0) {
    const long long now = sw_now();
    if (t0 == 0) t0 = now;
    if (now - t0 > sh->wait_ns) *(volatile int *)&sh->failed = 1;
    return sw_failed(sh) ? 0 : t0;
}

// Waits of a whole warp for phase `parity` of bar, with one answer for all its
// lanes: the warp's next __syncwarp has them all or none.  false: the wait gave
// up, and the warp leaves the run without an arrival: the level mbarriers may
// be in an earlier phase, where a wait returns at once and an arrival for more
// than is pending is an error.  The vote costs 1 % (2048^2 natural FP64 2.40 ms
// against 2.37); letting a warp go on without one and keeping back its arrivals
// cost more (2.42 and 2.51).  The threads sleep in mbarrier.try_wait: polling
// with test_wait took issue slots from the groups at work (512^2 natural FP64
// 260 us against 223).
__device__ __forceinline__ bool sw_wait(SweepShared *sh, unsigned long long *bar, unsigned parity) {
    long long t0 = 0;
#pragma unroll 1
    for (int i = 1;; ++i) {
        if (__all_sync(kWarp, mbar_try_wait(as_bar(bar), parity))) return true;
        if (i % kPolls == 0) {
            t0 = sw_patience(sh, t0);
            if (__any_sync(kWarp, t0 == 0)) return false;
        }
    }
}

// The same for one lane.
__device__ __forceinline__ bool sw_wait_lane(SweepShared *sh, unsigned long long *bar, unsigned parity) {
    long long t0 = 0;
#pragma unroll 1
    for (int i = 1;; ++i) {
        if (mbar_try_wait(as_bar(bar), parity)) return true;
        if (i % kPolls == 0) {
            t0 = sw_patience(sh, t0);
            if (t0 == 0) return false;
        }
    }
}

// Until an issued copy has arrived, whatever else gave up.
__device__ __forceinline__ void sw_drain(unsigned long long *bar, unsigned parity) {
    const long long t0 = sw_now();
    while (!mbar_try_wait(as_bar(bar), parity) && sw_now() - t0 < kDrainNs) {
    }
}

// The copying warps take the run's records in turn, each once the records
// whose room it needs are given back.  Issuing a record is a chain of about 500
// cycles whatever its size, which with one warp held a run of wide levels to
// 36 GB/s; so there are kCopyWarps of them.  Returns when the warp's copies have
// arrived.
__device__ __forceinline__ void sw_copy(SweepShared *sh, unsigned stage, const Record *__restrict__ recs, int n_rec,
                                        int base, const unsigned char *__restrict__ blob,
                                        const unsigned char *__restrict__ bp, int vbytes, int warp) {
    const int lane = threadIdx.x & 31;
    int4 a = make_int4(0, 0, 0, 0), b = a;
    auto fetch = [&](int i) {
        if (i < n_rec) {
            a = *reinterpret_cast<const int4 *>(recs + i);
            b = *(reinterpret_cast<const int4 *>(recs + i) + 1);
        }
    };
    bool good = true;  // no wait has given up, here or elsewhere: after one, no further copy is issued
    int last = -1;     // the warp's last record issued
    fetch(kCopyWarps * lane + warp);
#pragma unroll 1
    for (int i0 = warp; i0 < n_rec && good; i0 += 32 * kCopyWarps) {
        const int4 ca = a, cb = b;
        fetch(i0 + kCopyWarps * (32 + lane));
#pragma unroll 1
        for (int j = 0; j < 32 && i0 + kCopyWarps * j < n_rec && good; ++j) {
            const int i = base + i0 + kCopyWarps * j;
            if (lane == j) {
#pragma unroll 1
                for (int f = base + cb.z; f < base + cb.y && good; ++f)
                    good = sw_wait_lane(sh, &sh->empty[f % kSlots], (unsigned)(f / kSlots) & 1u);
                good = good && !sw_failed(sh);
                if (good) {
                    unsigned long long *bar = &sh->full[i % kSlots];
                    mbar_arrive_expect_tx(as_bar(bar), (unsigned)(ca.y + ca.w));
                    bulk_copy(stage + cb.x, blob + (int64_t)ca.x * 16, (unsigned)ca.y, bar);
                    if (ca.w)
                        bulk_copy(stage + cb.x + ca.y, bp + (int64_t)ca.z * vbytes, (unsigned)ca.w, bar);
                }
            }
            good = __shfl_sync(0xffffffffu, good, j);
            if (good) last = i;
        }
    }
    // none of the warp's copies in flight: those before the last kSlots records were used
#pragma unroll 1
    for (int i = last; i >= base && i > last - kSlots; i -= kCopyWarps)
        sw_drain(&sh->full[i % kSlots], (unsigned)(i / kSlots) & 1u);
}

// A chunk's header.
struct ChunkView {
    int pos, m, wf, next;  // wf: width << kFlagBits | flags
    int boff, level, next_rec, rec_arrive;
    __device__ __forceinline__ int mp() const { return (m + 3) & ~3; }
};

__device__ __forceinline__ ChunkView sw_view(const unsigned char *stage, int at) {
    const int4 h0 = *reinterpret_cast<const int4 *>(stage + at);
    const int4 h1 = *reinterpret_cast<const int4 *>(stage + at + 16);
    return ChunkView{h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
}
// the rest of it, needed less often
__device__ __forceinline__ int sw_level_arrive(const unsigned char *stage, int at) {
    return *reinterpret_cast<const int *>(stage + at + 32);
}
__device__ __forceinline__ int sw_blob_offset(const unsigned char *stage, int at) {
    return *reinterpret_cast<const int *>(stage + at + 36);
}

// One row's operands (of wider rows: right-hand side and diagonal).  W: 2 or 3,
// the chunk's layout; 0: whatever its header says.
template <typename VT> struct RowOps {
    VT b, d, v0, v1, v2;
    int s0, s1, s2;
};

template <typename VT, int W>
__device__ __forceinline__ void sw_load(const unsigned char *stage, int at, const ChunkView &c, int t, RowOps<VT> &R) {
    if (t >= c.m || (W == 0 && (c.wf & kDirect))) return;
    const unsigned char *data = stage + at + kHeader;
    R.b = reinterpret_cast<const VT *>(stage + c.boff)[t];
    if (W == 2 || (W == 0 && (c.wf & kTwo))) {
        if constexpr (sizeof(VT) == 8) {
            const double2 q0 = reinterpret_cast<const double2 *>(data)[t];
            const int4 q1 = reinterpret_cast<const int4 *>(data)[c.mp() + t];
            R.v0 = q0.x;
            R.v1 = q0.y;
            R.d = __hiloint2double(q1.y, q1.x);
            R.s0 = q1.z;
            R.s1 = q1.w;
        } else {
            const int4 q = reinterpret_cast<const int4 *>(data)[t];
            R.v0 = __int_as_float(q.x);
            R.v1 = __int_as_float(q.y);
            R.s0 = q.z;
            R.s1 = q.w;
            R.d = reinterpret_cast<const float *>(data + c.mp() * 16)[t];
        }
    } else if (W == 3 || (W == 0 && (c.wf & kThree))) {
        int4 q;
        if constexpr (sizeof(VT) == 8) {
            const double2 q0 = reinterpret_cast<const double2 *>(data)[t];
            const double2 q1 = reinterpret_cast<const double2 *>(data)[c.mp() + t];
            q = reinterpret_cast<const int4 *>(data)[2 * c.mp() + t];
            R.v0 = q0.x;
            R.v1 = q0.y;
            R.v2 = q1.x;
            R.d = q1.y;
        } else {
            const float4 q0 = reinterpret_cast<const float4 *>(data)[t];
            q = reinterpret_cast<const int4 *>(data)[c.mp() + t];
            R.v0 = q0.x;
            R.v1 = q0.y;
            R.v2 = q0.z;
            R.d = q0.w;
        }
        R.s0 = q.x;
        R.s1 = q.y;
        R.s2 = q.z;
    } else {
        R.d = reinterpret_cast<const VT *>(data)[(c.wf >> kFlagBits) * c.mp() + t];
    }
}

// the solution a code names: a byte offset into the ring, or (negative) a position of x
template <typename VT>
__device__ __forceinline__ VT sw_solution(int code, const unsigned char *ring, const VT *xp) {
    return code >= 0 ? *reinterpret_cast<const VT *>(ring + code) : xp[~code];
}
template <typename VT> __device__ __forceinline__ VT sw_ring(int code, const unsigned char *ring) {
    return *reinterpret_cast<const VT *>(ring + code);
}

// the solution x of row t of a chunk
template <typename VT>
__device__ __forceinline__ void sw_store(const ChunkView &c, int t, VT x, unsigned char *ring, VT *xp) {
    const int p = c.pos + t;
    *reinterpret_cast<VT *>(ring + (p & (kRing - 1)) * (int)sizeof(VT)) = x;
    xp[p] = x;
}

// Sum of a row too wide for the stage, from the blob, eight entries in flight.
// A function of its own, for its registers.
template <typename VT>
__device__ __noinline__ VT sw_sum_direct(const unsigned char *__restrict__ data, int w, int mp, int t, const VT *xp) {
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned char *ring = smem + kSharedBytes;
    const VT *pv = reinterpret_cast<const VT *>(data) + t;
    const int *ps = reinterpret_cast<const int *>(data + (int64_t)(w + 1) * mp * (int)sizeof(VT)) + t;
    VT sum = VT(0);
    constexpr int U = 8;
    int i = 0;
#pragma unroll 1
    for (; i + U <= w; i += U, pv += (int64_t)U * mp, ps += (int64_t)U * mp) {
        VT v[U], x[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            v[q] = pv[(int64_t)q * mp];
            x[q] = sw_solution<VT>(ps[(int64_t)q * mp], ring, xp);
        }
#pragma unroll
        for (int q = 0; q < U; ++q) sum += v[q] * x[q];
    }
#pragma unroll 1
    for (; i < w; ++i, pv += mp, ps += mp) sum += *pv * sw_solution<VT>(*ps, ring, xp);
    return sum;
}

// sum of the entries' products of row t of a chunk of wider rows
template <typename VT>
__device__ VT sw_sum_any(const unsigned char *stage, int at, const ChunkView &c, int t, const RowOps<VT> &R,
                         const unsigned char *ring, const VT *xp, const unsigned char *__restrict__ blob) {
    VT sum = VT(0);
    const int w = c.wf >> kFlagBits;
    if (c.wf & kDirect)
        return sw_sum_direct<VT>(blob + (int64_t)sw_blob_offset(stage, at) * 16 + kHeader, w, c.mp(), t, xp);
    const VT *pv = reinterpret_cast<const VT *>(stage + at + kHeader);
    const int *ps = reinterpret_cast<const int *>(pv + (w + 1) * c.mp());
    // four entries at a time: their solutions are read before any is used
    constexpr int U = 4;
#pragma unroll 1
    for (int i = 0; i < w; i += U) {
        VT v[U], x[U];
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (i + q < w) {
                v[q] = pv[(i + q) * c.mp() + t];
                x[q] = sw_solution<VT>(ps[(i + q) * c.mp() + t], ring, xp);
            }
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (i + q < w) sum += v[q] * x[q];
    }
    return sum;
}

// Rows a thread of a group solves in one chunk: two on the largest groups
// (2048^2 natural FP64 3.37 ms against 3.65 with one, 512^2 FP32 248 us against 297).
template <int T> constexpr int group_rows() { return T == 128 ? 2 : 1; }

// This thread's RW rows (t, t + T, ...) of a chunk of layout W (2 or 3).  RING:
// all its solutions are in the ring.  The rows' sums are independent chains:
// only the reads and the stores ask whether a row exists.
template <typename VT, int T, bool DIV, int W, int RW, bool RING>
__device__ __forceinline__ void sw_rows(const ChunkView &c, int t, const RowOps<VT> (&R)[RW], unsigned char *ring,
                                        VT *xp) {
    VT x[RW][3];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        x[r][0] = RING ? sw_ring<VT>(R[r].s0, ring) : sw_solution<VT>(R[r].s0, ring, xp);
        x[r][1] = RING ? sw_ring<VT>(R[r].s1, ring) : sw_solution<VT>(R[r].s1, ring, xp);
        if (W == 3) x[r][2] = RING ? sw_ring<VT>(R[r].s2, ring) : sw_solution<VT>(R[r].s2, ring, xp);
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        VT sum = VT(0);
        sum += R[r].v0 * x[r][0];
        sum += R[r].v1 * x[r][1];
        if (W == 3) sum += R[r].v2 * x[r][2];
        x[r][0] = finish_row<VT, DIV>(R[r].b, sum, R[r].d);
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
        if (t + r * T < c.m) sw_store<VT>(c, t + r * T, x[r][0], ring, xp);
}

// Row t of any other chunk.
template <typename VT, bool DIV>
__device__ __forceinline__ void sw_row_any(const unsigned char *stage, int at, const ChunkView &c, int t,
                                           RowOps<VT> &R, unsigned char *ring, VT *xp,
                                           const unsigned char *__restrict__ blob, const VT *__restrict__ bp) {
    if (t >= c.m) return;
    const VT sum = sw_sum_any<VT>(stage, at, c, t, R, ring, xp, blob);
    if (c.wf & kDirect) {
        R.b = bp[c.pos + t];
        R.d = reinterpret_cast<const VT *>(blob + (int64_t)sw_blob_offset(stage, at) * 16 +
                                           kHeader)[(int64_t)(c.wf >> kFlagBits) * c.mp() + t];
    }
    sw_store<VT>(c, t, finish_row<VT, DIV>(R.b, sum, R.d), ring, xp);
}

__device__ __forceinline__ void sw_arrive(unsigned long long *bar, int count) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// The wait for the level before.
__device__ __forceinline__ bool sw_wait_before(SweepShared *sh, const ChunkView &c, int level0) {
    if (c.level == 0) return true;
    const int l = level0 + c.level - 1;
    return sw_wait(sh, &sh->level[l % kLevels], (unsigned)(l / kLevels) & 1u);
}

// Chunk c of layout W for a group: operands, the wait for the level before, RW
// rows a thread, the arrivals.  T threads a group, t the thread's rank.
template <typename VT, int T, bool DIV, int W, int RW, bool RING = true>
__device__ __forceinline__ bool sw_chunk(SweepShared *sh, unsigned char *ring, const unsigned char *stage, int at,
                                         const ChunkView &c, int t, int rec, int level0, VT *xp) {
    const bool first = (threadIdx.x & 31) == 0;  // of its warp
    RowOps<VT> R[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        R[r].b = R[r].v0 = R[r].v1 = R[r].v2 = VT(0);  // of a row that is not there
        R[r].d = VT(1);
        R[r].s0 = R[r].s1 = R[r].s2 = kRing * (int)sizeof(VT);
        sw_load<VT, W>(stage, at, c, t + r * T, R[r]);
    }
    const int owed = sw_level_arrive(stage, at);
    // the operands are in registers: the record's room may be reused
    __syncwarp();
    if (first) sw_arrive(&sh->empty[rec % kSlots], c.rec_arrive);
    if (!sw_wait_before(sh, c, level0)) return false;
    sw_rows<VT, T, DIV, W, RW, RING>(c, t, R, ring, xp);
    __syncwarp();
    if (first) sw_arrive(&sh->level[(level0 + c.level) % kLevels], owed);
    return true;
}

// Any other chunk: a function of its own, so that its registers are not added
// to those of the common layouts.
template <typename VT, int T, bool DIV>
__device__ __noinline__ bool sw_chunk_any(int at, int t, int rec, int level0, VT *xp, const unsigned char *blob,
                                          const VT *bp) {
    extern __shared__ __align__(128) unsigned char smem[];
    SweepShared *sh = reinterpret_cast<SweepShared *>(smem);
    unsigned char *ring = smem + kSharedBytes;
    const unsigned char *stage = smem + kSharedBytes + ring_bytes<VT>();
    const ChunkView c = sw_view(stage, at);
    const bool first = (threadIdx.x & 31) == 0;  // of its warp
    if (c.wf & kTwo) return sw_chunk<VT, T, DIV, 2, group_rows<T>(), false>(sh, ring, stage, at, c, t, rec, level0, xp);
    if (c.wf & kThree) return sw_chunk<VT, T, DIV, 3, group_rows<T>(), false>(sh, ring, stage, at, c, t, rec, level0, xp);
    RowOps<VT> R;
    sw_load<VT, 0>(stage, at, c, t, R);
    if (!sw_wait_before(sh, c, level0)) return false;
    sw_row_any<VT, DIV>(stage, at, c, t, R, ring, xp, blob, bp);
    const int owed = sw_level_arrive(stage, at);
    __syncwarp();
    if (first) {
        sw_arrive(&sh->level[(level0 + c.level) % kLevels], owed);
        sw_arrive(&sh->empty[rec % kSlots], c.rec_arrive);
    }
    return true;
}

// Sweeps one run with kGroups groups of T solving threads and kCopyWarps
// copying warps.  rec0, level0: records and levels this CTA has seen before (the
// mbarriers' phases go on from there).  Chunks are taken in turn, so the
// first unsolved one always has what it waits for: its level's predecessor is
// solved, and its record's room was given back by chunks before it.
template <typename VT, int T, bool DIV>
__device__ void sw_run(const SweepPack::Run &run, const Record *__restrict__ recs,
                       const unsigned char *__restrict__ blob, const VT *__restrict__ bp, VT *xp, unsigned char *smem,
                       int rec0, int level0) {
    SweepShared *sh = reinterpret_cast<SweepShared *>(smem);
    unsigned char *ring = smem + kSharedBytes;
    const unsigned char *stage = smem + kSharedBytes + ring_bytes<VT>();
    if (threadIdx.x >= kGroups * T) {
        sw_copy(sh, smem_u32(stage), recs + run.rec0, run.n_rec, rec0, blob,
                reinterpret_cast<const unsigned char *>(bp), (int)sizeof(VT), (int)(threadIdx.x - kGroups * T) / 32);
    } else {
        const int g = threadIdx.x / T, t = threadIdx.x % T;
        int at = run.at[g], rec = rec0 + run.rec[g];
        bool good = true;
#pragma unroll 1
        while (at >= 0 && good) {
            good = sw_wait(sh, &sh->full[rec % kSlots], (unsigned)(rec / kSlots) & 1u);
            if (!good) break;
            const ChunkView c = sw_view(stage, at);
            const int kind = c.wf & (kTwo | kThree | kRingOnly);
            constexpr int RW = group_rows<T>();
            if (kind == (kTwo | kRingOnly)) {
                if (RW == 1 || c.m <= T) good = sw_chunk<VT, T, DIV, 2, 1>(sh, ring, stage, at, c, t, rec, level0, xp);
                else good = sw_chunk<VT, T, DIV, 2, RW>(sh, ring, stage, at, c, t, rec, level0, xp);
            } else if (kind == (kThree | kRingOnly)) {
                if (RW == 1 || c.m <= T) good = sw_chunk<VT, T, DIV, 3, 1>(sh, ring, stage, at, c, t, rec, level0, xp);
                else good = sw_chunk<VT, T, DIV, 3, RW>(sh, ring, stage, at, c, t, rec, level0, xp);
            } else {
                good = sw_chunk_any<VT, T, DIV>(at, t, rec, level0, xp, blob, bp);
            }
            at = c.next;
            rec = rec0 + c.next_rec;
        }
    }
    __syncthreads();
}

// After a wait that gave up: no number in place of a solution.
template <typename VT> __device__ __forceinline__ void sw_no_solution(const SweepPack::Run &run, VT *xp) {
#pragma unroll 1
    for (int p = run.pos0 + threadIdx.x; p < run.pos1; p += blockDim.x) xp[p] = VT(NAN);
}

// level_arrivals, rec_arrivals: what completes a level and gives a record back
template <typename VT>
__device__ __forceinline__ void sw_init(unsigned char *smem, int level_arrivals, int rec_arrivals, const SweepWait &wait) {
    SweepShared *sh = reinterpret_cast<SweepShared *>(smem);
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(as_bar(&sh->full[i]), 1);
            mbar_init(as_bar(&sh->empty[i]), rec_arrivals);
        }
        for (int i = 0; i < kLevels; ++i) mbar_init(as_bar(&sh->level[i]), level_arrivals + (wait.never ? 1 : 0));
        sh->wait_ns = wait.ns;
        sh->failed = 0;
        mbar_fence_init();
        reinterpret_cast<VT *>(smem + kSharedBytes)[kRing] = VT(0);  // the slot of padding
    }
}

// CTA v sweeps the run for right-hand side v
template <typename VT, int T, bool DIV>
__global__ void __launch_bounds__(kGroups * T + 32 * kCopyWarps, 1)
    sweep_kernel(const SweepPack::Run run, const Record *__restrict__ recs, const unsigned char *__restrict__ blob,
                 int64_t npos, const VT *__restrict__ bp, VT *xp, DevStatus *status, const SweepWait wait) {
    extern __shared__ __align__(128) unsigned char smem[];
    sw_init<VT>(smem, run.level_chunks * (T / 32), kRecChunks * (T / 32), wait);
    __syncthreads();
    bp += blockIdx.x * npos;
    xp += blockIdx.x * npos;
    sw_run<VT, T, DIV>(run, recs, blob, bp, xp, smem, 0, 0);
    if (*(volatile int *)&reinterpret_cast<SweepShared *>(smem)->failed) {
        if (threadIdx.x == 0 && status) report(status, SMAX_ERR_TIMEOUT, run.pos0);
        sw_no_solution<VT>(run, xp);
    }
}

// CTAs take matrices (one run each) from a work queue
template <typename VT, int T>
__global__ void __launch_bounds__(kGroups * T + 32 * kCopyWarps, T <= 32 ? 2 : 1)
    sweep_batch_kernel(const SweepPack::Run *__restrict__ runs, const int *__restrict__ queue_order, int n_mats,
                       int *queue, const Record *__restrict__ recs, const unsigned char *__restrict__ blob,
                       const VT *__restrict__ bp, VT *xp, int *status, const SweepWait wait) {
    extern __shared__ __align__(128) unsigned char smem[];
    SweepShared *sh = reinterpret_cast<SweepShared *>(smem);
    sw_init<VT>(smem, runs[0].level_chunks * (T / 32), kRecChunks * (T / 32), wait);
    // what the CTA keeps from one matrix to the next is in shared memory: the
    // sweep needs the registers
    volatile SweepShared *vs = sh;
    if (threadIdx.x == 0) vs->rec0 = vs->level0 = 0;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int q = atomicAdd(queue, 1);
            vs->mat = q < n_mats ? queue_order[q] : -1;
        }
        __syncthreads();
        if (vs->mat < 0) return;
        if (!vs->failed) sw_run<VT, T, false>(runs[vs->mat], recs, blob, bp, xp, smem, vs->rec0, vs->level0);
        const SweepPack::Run &run = runs[vs->mat];
        if (vs->failed) {
            if (threadIdx.x == 0) *(volatile int *)status = SMAX_ERR_TIMEOUT;
            sw_no_solution<VT>(run, xp);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            vs->rec0 = vs->rec0 + run.n_rec;
            vs->level0 = vs->level0 + run.n_levels;
        }
    }
}

// stage bytes of a CTA: an SM has 227 KB of shared memory for one CTA, 113 KB for each of two
int sweep_stage_bytes(int vbytes, bool shared_sm) {
    const int ring = vbytes == 8 ? ring_bytes<double>() : ring_bytes<float>();
    return ((shared_sm ? 113 : 227) * 1024 - ring - kSharedBytes) / 128 * 128;
}

size_t sweep_smem(const SweepPack &pk) {
    return kSharedBytes + (pk.vbytes == 8 ? ring_bytes<double>() : ring_bytes<float>()) + pk.stage_bytes;
}

// the shared-memory opt-in of every sweep kernel, set when a pack is built and
// not inside a capture
template <typename VT, int T> void set_attr_t(int bytes) {
    SMAX_CUDA(cudaFuncSetAttribute(sweep_batch_kernel<VT, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    SMAX_CUDA(cudaFuncSetAttribute(sweep_kernel<VT, T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    SMAX_CUDA(cudaFuncSetAttribute(sweep_kernel<VT, T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}
template <typename VT> void set_attr() {
    const int bytes = kSharedBytes + ring_bytes<VT>() + sweep_stage_bytes(sizeof(VT), false);
    set_attr_t<VT, 32>(bytes);
    set_attr_t<VT, 64>(bytes);
    set_attr_t<VT, 128>(bytes);
}

// Threads of a group: a row a thread at the run's widest level, at most 128 of
// up to two rows (wider levels are several chunks).
int group_threads(int max_rows) { return max_rows <= 32 ? 32 : (max_rows <= 64 ? 64 : 128); }

template <typename VT, bool DIV>
void launch_run(const SweepPack &pk, const SweepPack::Run &run, int threads, int64_t k, const VT *bp, VT *xp,
                DevStatus *status, const SweepWait &wait, cudaStream_t st) {
    const size_t sm = sweep_smem(pk);
    const Record *recs = pk.recs.as<Record>();
    const unsigned char *blob = pk.blob.as<unsigned char>();
    auto go = [&](auto kern, int t) {
        kern<<<(unsigned)k, kGroups * t + 32 * kCopyWarps, sm, st>>>(run, recs, blob, pk.npos, bp, xp, status, wait);
    };
    if (threads == 32) go(sweep_kernel<VT, 32, DIV>, 32);
    else if (threads == 64) go(sweep_kernel<VT, 64, DIV>, 64);
    else go(sweep_kernel<VT, 128, DIV>, 128);
}

}  // namespace

bool build_sweep_pack(SweepPack &pk, const int *rp, const int *ci, const void *val, const void *D, int vbytes,
                      int64_t n, const int *order, const std::vector<int> &src_begin, const std::vector<int> &count,
                      const std::vector<SweepStep> &steps, bool div, bool batch, cudaStream_t st) {
    const int L = (int)count.size();
    if ((int)src_begin.size() != L) fail(SMAX_ERR_STATE, "inconsistent sweep steps");
    pk = SweepPack();
    pk.n = n;
    pk.vbytes = vbytes;
    pk.div = div;
    // a batch sweeps all its runs in one launch: one CTA size, and two CTAs on
    // an SM when there are more matrices than SMs and the CTAs are small enough
    int batch_threads = 0, n_runs = 0;
    for (const SweepStep &step : steps)
        if (step.kind == 1) {
            ++n_runs;
            for (int s = step.first; s < step.first + step.count; ++s)
                batch_threads = std::max(batch_threads, group_threads(count[s]));
        }
    pk.shared_sm = batch && n_runs > sm_count() && batch_threads <= 32;
    pk.stage_bytes = sweep_stage_bytes(vbytes, pk.shared_sm);
    if (vbytes == 8) set_attr<double>();
    else set_attr<float>();
    int64_t rows = 0;
    for (int s = 0; s < L; ++s) rows += count[s];
    if (rows != n) fail(SMAX_ERR_STATE, "sweep steps do not cover all rows");
    if (n == 0 || L == 0) return true;
    // the widest row of every level
    std::vector<int> w(L);
    int h_end = 0;
    {
        DevBuf len(sizeof(int) * n), wmax(sizeof(int) * L), d_beg(sizeof(int) * L), d_end(sizeof(int) * L);
        std::vector<int> end(L);
        for (int s = 0; s < L; ++s) end[s] = src_begin[s] + count[s];
        SMAX_CUDA(cudaMemcpyAsync(d_beg.p, src_begin.data(), sizeof(int) * L, cudaMemcpyHostToDevice, st));
        SMAX_CUDA(cudaMemcpyAsync(d_end.p, end.data(), sizeof(int) * L, cudaMemcpyHostToDevice, st));
        sw_off_len_kernel<<<grid_for(n), 256, 0, st>>>(rp, order, n, len.as<int>());
        SMAX_CUDA(cudaGetLastError());
        size_t tb = 0;
        SMAX_CUDA(cub::DeviceSegmentedReduce::Max(nullptr, tb, len.as<int>(), wmax.as<int>(), L, d_beg.as<int>(),
                                                  d_end.as<int>(), st));
        DevBuf tmp(tb);
        SMAX_CUDA(cub::DeviceSegmentedReduce::Max(tmp.p, tb, len.as<int>(), wmax.as<int>(), L, d_beg.as<int>(),
                                                  d_end.as<int>(), st));
        SMAX_CUDA(cudaMemcpyAsync(w.data(), wmax.p, sizeof(int) * L, cudaMemcpyDeviceToHost, st));
        SMAX_CUDA(cudaMemcpyAsync(&h_end, rp + n, sizeof(int), cudaMemcpyDeviceToHost, st));
        SMAX_CUDA(cudaStreamSynchronize(st));
    }
    long long padded = 0;
    for (int s = 0; s < L; ++s) {
        w[s] = count[s] > 0 ? std::max(w[s], 0) : 0;
        padded += (long long)count[s] * w[s];
        if (w[s] >= (1 << 20)) return false;
    }
    const long long off_diag = (long long)h_end - n;
    if (padded > 3 * off_diag + (1ll << 20) || padded >= (1ll << 31) - (1ll << 26)) return false;

    // --- chunks, records and the stage schedule
    std::vector<ChunkDesc> ch;
    std::vector<int> ch_src;
    std::vector<Record> recs;
    std::vector<std::pair<int, int>> run_chunks;  // chunks of each run
    const int vb = vbytes, S = pk.stage_bytes;
    // records of an eighth of the stage: 2048^2 natural FP64 2.46 ms; a sixteenth
    // 3.37 (a copy costs its issue), a tenth 3.11, a fifth 2.47
    const int chunk_cap = S / 6 / 16 * 16, rec_cap = S / 8 / 16 * 16;
    int64_t off = 0, pos = 0;  // blob bytes, positions
    bool wraps = false;
    auto add_chunk = [&](int s, int t0, int m, int lpos, int lend, int rpos, int flags, int level,
                         int pad = 4) {
        ChunkDesc d{};
        d.pos = (int)pos;
        d.m = m;
        d.w = w[s];
        d.mp = (m + pad - 1) / pad * pad;
        d.off = (int)(off / 16);
        d.lpos = lpos;
        d.lend = lend;
        d.rpos = rpos;
        d.flags = flags;
        d.level = level;
        d.next = -1;
        ch.push_back(d);
        ch_src.push_back(src_begin[s] + t0);
        pos += d.mp;
        off += kHeader + (int64_t)d.mp * row_bytes(flags, w[s], vb);
    };
    for (const SweepStep &step : steps) {
        if (step.kind == 0) {
            for (int s = step.first; s < step.first + step.count; ++s) {
                if (count[s] == 0) continue;
                const int p0 = (int)pos;
                off = (off + kHeader + 127) / 128 * 128 - kHeader;  // columns of whole cache lines
                add_chunk(s, 0, count[s], p0, p0 + count[s], p0, 0, 0, 32);
                const ChunkDesc &d = ch.back();
                pk.items.push_back({true, (int)pk.wides.size(), 0});
                pk.wides.push_back({d.pos, d.m, d.w, d.mp, d.off});
            }
            continue;
        }
        SweepPack::Run run{};
        run.rec0 = (int)recs.size();
        run.pos0 = (int)pos;
        const int c_run = (int)ch.size(), rpos = (int)pos;
        int widest = 0;
        for (int s = step.first; s < step.first + step.count; ++s) widest = std::max(widest, count[s]);
        const int T = batch ? batch_threads : group_threads(widest);
        for (int s = step.first; s < step.first + step.count; ++s) {
            const int m = count[s];
            if (m == 0) continue;
            wraps = wraps || m > kRing - 4;
            // a level near the waits' limit (an entry after the other in its rows,
            // and what the SM takes in) is left to the plain kernels
            if (25ll * w[s] * (m / (kGroups * T) + 1) + (long long)m * w[s] / 4 > kLevelTime) return false;
            const int layout = w[s] <= 2 ? kTwo : (w[s] == 3 ? kThree : 0);
            const long long each = (long long)row_bytes(layout, w[s], vb) + vb;  // with its right-hand side
            // two rows a thread, but one where a division each is the longest part
            // of a level that the groups can share: 8 right-hand sides, 400^2
            // 432 us (two rows: 469); 32 of 1024^2 1.51 ms with two rows
            // where a level has more rows than the CTA threads, 1.76 without
            const int T_rows = T < 128 || layout == 0 || (div && m <= 4 * T) ? T : T * group_rows<128>();
            const long long fit = std::min<long long>((chunk_cap - kHeader) / each, T_rows) / 4 * 4;
            if (fit < 4) {
                // in place, as many rows at a time as the threads hold
                const int lpos = (int)pos, lend = lpos + (m + 3) / 4 * 4, per = T;
                for (int t0 = 0; t0 < m; t0 += per)
                    add_chunk(s, t0, std::min(per, m - t0), lpos, lend, rpos, kDirect, run.n_levels);
                ++run.n_levels;
                continue;
            }
            int per = m;
            if (m > fit) {
                const int parts = (int)((m + fit - 1) / fit);
                per = (m + parts - 1) / parts;
                per = std::min<long long>((per + 31) / 32 * 32, fit >= 32 ? fit / 32 * 32 : fit);
            }
            const int lpos = (int)pos;
            // the level's padded end: every chunk but the last holds a multiple of 4 rows
            const int lend = lpos + (m - 1) / per * per + ((m - 1) % per + 1 + 3) / 4 * 4;
            for (int t0 = 0; t0 < m; t0 += per)
                add_chunk(s, t0, std::min(per, m - t0), lpos, lend, rpos, layout, run.n_levels);
            ++run.n_levels;
        }
        run.pos1 = (int)pos;
        const int c_end = (int)ch.size();
        // records: consecutive chunks up to rec_cap bytes, wide levels' rows read in place on their own
        std::vector<int> first_chunk;
        for (int c = c_run; c < c_end; ++c) {
            const bool direct = ch[c].flags & kDirect;
            const int bytes = direct ? kHeader : kHeader + ch[c].mp * row_bytes(ch[c].flags, ch[c].w, vb);
            const int bbytes = direct ? 0 : ch[c].mp * vb;
            const bool open = c > c_run && !direct && !(ch[c - 1].flags & kDirect) &&
                              c - first_chunk.back() < kRecChunks && recs.back().bytes + recs.back().bbytes + bytes + bbytes <= rec_cap;
            if (!open) {
                first_chunk.push_back(c);
                recs.push_back(Record{ch[c].off, 0, ch[c].pos, 0, 0, 0, 0, 0});
            }
            recs.back().bytes += bytes;
            recs.back().bbytes += bbytes;
        }
        run.n_rec = (int)recs.size() - run.rec0;
        first_chunk.push_back(c_end);
        // where records lie: round the stage, each after the one before; a record
        // waits for the latest earlier one whose room it takes, and for all but
        // the kWindow - 1 before it.  A group's next chunk is at most kGroups
        // records ahead of the one it has solved, so the mbarrier it then polls
        // has completed every phase but the one it waits for
        int cursor = 0;
        Record *r = recs.data() + run.rec0;
        for (int i = 0; i < run.n_rec; ++i) {
            const int z = r[i].bytes + r[i].bbytes;
            if (cursor + z > S) cursor = 0;
            r[i].stage = cursor;
            cursor += z;
            r[i].dep = std::max(0, i - kWindow + 1);
            for (int j = i - 1; j >= r[i].dep; --j) {
                const int zj = r[j].bytes + r[j].bbytes;
                if (r[j].stage < r[i].stage + z && r[i].stage < r[j].stage + zj) {
                    r[i].dep = j + 1;
                    break;
                }
            }
            if (i > 0) r[i].dep = std::max(r[i].dep, r[i - 1].dep);
            r[i].from = i >= kCopyWarps ? r[i - kCopyWarps].dep : 0;  // waited for by the same warp
        }
        // stage offsets; arrivals: every warp of a chunk's group owes its record
        // and its level one, the last chunk of a record the rest of kRecChunks
        // and the last of a level the rest of the most chunks a level has
        std::vector<int> where(c_end - c_run), rec_of(c_end - c_run);
        for (int i = 0; i < run.n_rec; ++i)
            for (int c = first_chunk[i]; c < first_chunk[i + 1]; ++c) {
                ChunkDesc &d = ch[c];
                d.boff = c > first_chunk[i] ? ch[c - 1].boff + ch[c - 1].mp * vb : r[i].stage + r[i].bytes;
                where[c - c_run] = r[i].stage + (int)(((int64_t)d.off - r[i].off) * 16);
                rec_of[c - c_run] = i;
                d.rec_arrive = c + 1 < first_chunk[i + 1] ? 1 : kRecChunks - (c - first_chunk[i]);
            }
        for (int c = c_run, in_level = 0; c < c_end; ++c) {
            ++in_level;
            if (c + 1 < c_end && ch[c + 1].level == ch[c].level) continue;
            if (in_level > kMaxArrivals / (T / 32)) return false;  // tens of millions of rows: the plain kernels
            run.level_chunks = std::max(run.level_chunks, in_level);
            ch[c].lev_arrive = in_level;  // made good below
            in_level = 0;
        }
        for (int c = c_run; c < c_end; ++c) {
            const int n = c - c_run + kGroups;
            ch[c].next = n < c_end - c_run ? where[n] : -1;
            ch[c].next_rec = n < c_end - c_run ? rec_of[n] : 0;
        }
        for (int g = 0; g < kGroups; ++g) {
            run.at[g] = g < c_end - c_run ? where[g] : -1;
            run.rec[g] = g < c_end - c_run ? rec_of[g] : 0;
        }
        run_chunks.push_back({c_run, c_end});
        if (run.n_rec > 0) pk.items.push_back({false, (int)pk.runs.size(), T});
        pk.runs.push_back(run);
    }
    // a batch's mbarriers serve all its runs: one count
    int most = 1;
    for (const SweepPack::Run &run : pk.runs) most = std::max(most, run.level_chunks);
    for (size_t i = 0; i < pk.runs.size(); ++i) {
        if (batch || pk.runs[i].level_chunks == 0) pk.runs[i].level_chunks = most;
        for (int c = run_chunks[i].first; c < run_chunks[i].second; ++c)
            ch[c].lev_arrive = ch[c].lev_arrive > 0 ? pk.runs[i].level_chunks - ch[c].lev_arrive + 1 : 1;
    }
    if (pos >= (1ll << 31) - 8 || off / 16 >= (1ll << 31) - 8) return false;
    pk.npos = pos;
    pk.blob_bytes = off;
    pk.n_chunks = (int)ch.size();

    // --- device copies
    std::vector<int> pch(pos);
    for (int c = 0; c < pk.n_chunks; ++c) std::fill_n(pch.begin() + ch[c].pos, ch[c].mp, c);
    auto up = [&](DevBuf &d, const void *h, size_t bytes) {
        d.alloc(bytes ? bytes : 16);
        if (bytes) SMAX_CUDA(cudaMemcpyAsync(d.p, h, bytes, cudaMemcpyHostToDevice, st));
    };
    up(pk.pchunk, pch.data(), sizeof(int) * pos);
    up(pk.chunks, ch.data(), sizeof(ChunkDesc) * ch.size());
    up(pk.recs, recs.data(), sizeof(Record) * recs.size());
    up(pk.drun, pk.runs.data(), sizeof(SweepPack::Run) * pk.runs.size());
    DevBuf d_src, pos_of_row(sizeof(int) * n), glob(sizeof(int) * ch.size()), flag(sizeof(int));
    up(d_src, ch_src.data(), sizeof(int) * ch_src.size());
    pk.prow.alloc(sizeof(int) * pos);
    pk.blob.alloc((size_t)off);
    SMAX_CUDA(cudaMemsetAsync(pk.blob.p, 0, (size_t)off, st));
    SMAX_CUDA(cudaMemsetAsync(glob.p, 0, glob.bytes, st));
    SMAX_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
    const ChunkDesc *dch = pk.chunks.as<ChunkDesc>();
    sw_positions_kernel<<<grid_for(pos), 256, 0, st>>>(dch, d_src.as<int>(), pk.pchunk.as<int>(), order, pos,
                                                       pk.prow.as<int>(), pos_of_row.as<int>());
    auto fill = [&](auto zero) {
        using VT = decltype(zero);
        sw_fill_kernel<VT, true><<<grid_for(pos), 256, 0, st>>>(
            rp, ci, static_cast<const VT *>(val), static_cast<const VT *>(D), pos, pk.prow.as<int>(),
            pk.pchunk.as<int>(), pos_of_row.as<int>(), dch, pk.blob.as<unsigned char>(), div, wraps,
            glob.as<int>(), flag.as<int>());
    };
    if (vbytes == 8) fill(0.0);
    else fill(0.0f);
    sw_header_kernel<<<ceil_div_u(ch.size(), 256), 256, 0, st>>>(dch, pk.n_chunks, glob.as<int>(),
                                                                  pk.blob.as<unsigned char>());
    SMAX_CUDA(cudaGetLastError());
    int h_flag = 0;
    SMAX_CUDA(cudaMemcpyAsync(&h_flag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SMAX_CUDA(cudaStreamSynchronize(st));  // the temporaries die here
    pk.needs_x_init = h_flag != 0;
    sweep_reserve(pk, 1);
    return true;
}

void refill_sweep_pack(SweepPack &pk, const int *rp, const void *val, const void *D, cudaStream_t st) {
    if (pk.npos == 0) return;
    auto fill = [&](auto zero) {
        using VT = decltype(zero);
        sw_fill_kernel<VT, false><<<grid_for(pk.npos), 256, 0, st>>>(
            rp, nullptr, static_cast<const VT *>(val), static_cast<const VT *>(D), pk.npos, pk.prow.as<int>(),
            pk.pchunk.as<int>(), nullptr, pk.chunks.as<ChunkDesc>(), pk.blob.as<unsigned char>(), pk.div, false,
            nullptr, nullptr);
    };
    if (pk.vbytes == 8) fill(0.0);
    else fill(0.0f);
    SMAX_CUDA(cudaGetLastError());
}

void sweep_reserve(SweepPack &pk, int64_t k) {
    // right-hand sides solved at a time: one CTA each and one CTA per SM, and
    // at most 4 GiB of workspace
    const int64_t each = 2ll * pk.vbytes * std::max<int64_t>(1, pk.npos);
    k = std::max<int64_t>(1, std::min<int64_t>({k, sm_count(), (4ll << 30) / each, pk.most_vectors}));
    if (k <= pk.vectors) return;
    pk.vectors = 0;
    for (;; k = (k + 1) / 2) {
        try {
            pk.bp.ensure((size_t)(each / 2 * k));
            pk.xp.ensure((size_t)(each / 2 * k));
            break;
        } catch (const Error &e) {
            if (k == 1 || e.code != SMAX_ERR_OOM) throw;
            pk.bp.release();
            pk.xp.release();
            pk.most_vectors = (int)((k + 1) / 2);
        }
    }
    pk.vectors = (int)k;
}

template <typename VT>
void sweep_solve(const SweepPack &pk, const VT *B, VT *X, int64_t k, int64_t rs, int64_t vs, DevStatus *status,
                 const SweepWait &wait, cudaStream_t st) {
    if (pk.n == 0 || k == 0) return;
    if (pk.vectors < 1) fail(SMAX_ERR_STATE, "the sweep has no workspace");
    VT *bp = pk.bp.as<VT>(), *xp = pk.xp.as<VT>();
    const unsigned char *blob = pk.blob.as<unsigned char>();
    for (int64_t v0 = 0; v0 < k; v0 += pk.vectors) {
        const int64_t kv = std::min<int64_t>(pk.vectors, k - v0);
        const VT *Bv = B + v0 * vs;
        VT *Xv = X + v0 * vs;
        sw_gather<VT>(pk, Bv, Xv, kv, rs, vs, st);
        for (const SweepPack::Item &it : pk.items) {
            if (it.wide) {
                const SweepPack::Wide &L = pk.wides[it.index];
                const dim3 g(ceil_div_u(L.m, L.w > 2 * kWideEnts ? 64 : 256), (unsigned)kv);
                if (L.w > 2 * kWideEnts && pk.div) sw_wide_long_kernel<VT, true><<<g, 64, 0, st>>>(L, blob, pk.npos, bp, xp);
                else if (L.w > 2 * kWideEnts) sw_wide_long_kernel<VT, false><<<g, 64, 0, st>>>(L, blob, pk.npos, bp, xp);
                else if (pk.div) sw_wide_kernel<VT, true><<<g, 256, 0, st>>>(L, blob, pk.npos, bp, xp);
                else sw_wide_kernel<VT, false><<<g, 256, 0, st>>>(L, blob, pk.npos, bp, xp);
            } else if (pk.div) {
                launch_run<VT, true>(pk, pk.runs[it.index], it.threads, kv, bp, xp, status, wait, st);
            } else {
                launch_run<VT, false>(pk, pk.runs[it.index], it.threads, kv, bp, xp, status, wait, st);
            }
        }
        sw_scatter<VT>(pk, Xv, kv, rs, vs, st);
    }
    SMAX_CUDA(cudaGetLastError());
}

template <typename VT>
void sweep_solve_batch(const SweepPack &pk, const int *queue_order, int n_mats, int *queue, const VT *B, VT *X,
                       int *status, const SweepWait &wait, cudaStream_t st) {
    if (pk.n == 0 || n_mats == 0) return;
    VT *bp = pk.bp.as<VT>(), *xp = pk.xp.as<VT>();
    sw_gather<VT>(pk, B, X, 1, 1, 1, st);
    int threads = 32;
    for (const SweepPack::Item &it : pk.items) threads = std::max(threads, it.threads);
    const int ctas = std::max(1, std::min(n_mats, (pk.shared_sm ? 2 : 1) * sm_count()));
    SMAX_CUDA(cudaMemsetAsync(queue, 0, sizeof(int), st));
    const size_t sm = sweep_smem(pk);
    auto go = [&](auto kern, int t) {
        kern<<<ctas, kGroups * t + 32 * kCopyWarps, sm, st>>>(pk.drun.as<SweepPack::Run>(), queue_order, n_mats, queue, pk.recs.as<Record>(),
                                       pk.blob.as<unsigned char>(), bp, xp, status, wait);
    };
    if (threads == 32) go(sweep_batch_kernel<VT, 32>, 32);
    else if (threads == 64) go(sweep_batch_kernel<VT, 64>, 64);
    else go(sweep_batch_kernel<VT, 128>, 128);
    sw_scatter<VT>(pk, X, 1, 1, 1, st);
    SMAX_CUDA(cudaGetLastError());
}

template void sweep_solve<double>(const SweepPack &, const double *, double *, int64_t, int64_t, int64_t, DevStatus *,
                                  const SweepWait &, cudaStream_t);
template void sweep_solve<float>(const SweepPack &, const float *, float *, int64_t, int64_t, int64_t, DevStatus *,
                                 const SweepWait &, cudaStream_t);
template void sweep_solve_batch<double>(const SweepPack &, const int *, int, int *, const double *, double *,
                                        int *, const SweepWait &, cudaStream_t);
template void sweep_solve_batch<float>(const SweepPack &, const int *, int, int *, const float *, float *,
                                       int *, const SweepWait &, cudaStream_t);

}  // namespace smax
