// spmm.cu -- CRS SpMM Y = A X against a block of k dense vectors, sm_100a.
//
// Reference semantics: SPMM::CPU::naive_crs_spmm_row_maj / _col_maj
// (src/kernels/spmm/spmm_cpu/spmm_cpu_crs_impl.hpp:9-89).
//
// A row of a row-major block (X[col*k+v], Y[row*k+v]) is k contiguous values,
// read as 16-, 8- or 4-byte vectors, the widest that k and the addresses
// allow.  Two kernels, each summing a row's products in stored order:
//
// * spmm_group_kernel, the default.  G lanes share a row of A, NV vectors
//   each, for any G up to 32, so block widths that are no power of two keep
//   nearly all lanes busy.  One CTA per SM goes through a contiguous range of
//   rows (the rows of X that neighbouring rows share are still in its L1), and
//   a row's (col, val) pairs are in shared memory (cp.async) before they are
//   needed.  Bound by L1 wavefronts and the latency of the X rows.
// * spmm_row_major_kernel, a grid of all rows, for regular matrices where it
//   is the faster one (grid_suits).  Bound by L2 bandwidth when a row of X is
//   wide: it holds twice the warps.
//
// Column-major blocks are transposed into a row-major workspace (one pass over
// X) and run the group kernel, which writes Y column-major: A is read once
// and not once per vector.  The products per vector that it replaces spread a long
// row over the chip and add it up in slices.  So a row far longer than the
// others is not left to one group, which takes 0.1 us an entry, but cut into
// pieces, a warp each (spmm_piece_kernel, spmm_combine_kernel), and eight
// products at a time (four where a lane has four vectors) are added to a sum that
// loses less: 64 bits wide for FP32, compensated for FP64.  (Four at a time: rows of
// 900, k = 33 FP32 100 us, 87 with eight; sixteen in two plain sums lose more than
// the products do.)  (A row-major block is added up in stored order, by whichever
// kernel.)
//
// Measured before and after (before: the grid kernel, a warp per row for
// widths that are no power of two, k SpMVs for column-major blocks):
//   27-point 128^3, k = 16, FP64              652 -> 495 us
//   27-point 96^3, k = 5, FP64                560 -> 136 us
//   27-point 96^3, k = 8, column-major, FP64  688 -> 185 us
//   lognormal 600000 rows, k = 20, FP32       341 -> 183 us
//   lognormal 500000 rows, k = 16, FP64       569 -> 256 us
#include "spmv_formats.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

#include <cub/device/device_scan.cuh>

namespace smax {

namespace {

constexpr int kPiece = 128, kBigPiece = 512;  // entries of a piece, and of one of a row of over kPiece * 1024
__host__ __device__ constexpr int piece_size(int len) { return len > kPiece * 1024 ? kBigPiece : kPiece; }

template <typename VT> struct V16;
template <> struct V16<double> { using T = double2; static constexpr int N = 2; };
template <> struct V16<float> { using T = float4; static constexpr int N = 4; };

// One row of Y from its group of G lanes (lane g of the group, gmask the
// group's lanes): NV vectors of VEC values per lane, k == G * NV * VEC (VEC
// == 1 is the scalar path for k not divisible by the vector width).
template <typename VT, int G, int NV, int VEC>
__device__ __forceinline__ void spmm_row(int64_t row, int g, unsigned gmask, const int *__restrict__ row_ptr,
                                         const int *__restrict__ col, const VT *__restrict__ val, int64_t k,
                                         const VT *__restrict__ X, VT *__restrict__ Y) {
    VT acc[NV][VEC];
#pragma unroll
    for (int m = 0; m < NV; ++m)
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[m][i] = VT(0);
    const int s = row_ptr[row], e = row_ptr[row + 1];
    // FP32: the group's next G (col, val) pairs are loaded while the current
    // ones are used (k = 16 / 64 on the 27-point stencil: 7 % / 4 % faster);
    // FP64: the extra registers cost more occupancy than the overlap gains
    constexpr bool kAhead = sizeof(VT) == 4;
    int nc = 0;
    VT nv = VT(0);
    if (kAhead && s + g < e) {
        nc = ld_stream(col + s + g);
        nv = ld_stream(val + s + g);
    }
    for (int j0 = s; j0 < e; j0 += G) {
        const int jj = j0 + g;
        int myc;
        VT myv;
        if constexpr (kAhead) {
            myc = nc;
            myv = nv;
            nc = jj + G < e ? ld_stream(col + jj + G) : 0;
            nv = jj + G < e ? ld_stream(val + jj + G) : VT(0);
        } else {
            myc = jj < e ? ld_stream(col + jj) : 0;
            myv = jj < e ? ld_stream(val + jj) : VT(0);
        }
        const int cnt = min(G, e - j0);
        // unrolled so the X-row loads of consecutive entries overlap; holding
        // more rows in registers lowered occupancy and was measured slower
#pragma unroll 4
        for (int t = 0; t < cnt; ++t) {
            const int c = __shfl_sync(gmask, myc, t, G);
            const VT v = __shfl_sync(gmask, myv, t, G);
            const VT *xr = X + (int64_t)c * k;
#pragma unroll
            for (int m = 0; m < NV; ++m) {
                const int off = (m * G + g) * VEC;
                if constexpr (VEC == 2) {
                    const double2 xv = __ldg(reinterpret_cast<const double2 *>(xr + off));
                    acc[m][0] += v * xv.x;
                    acc[m][1] += v * xv.y;
                } else if constexpr (VEC == 4) {
                    const float4 xv = __ldg(reinterpret_cast<const float4 *>(xr + off));
                    acc[m][0] += v * xv.x;
                    acc[m][1] += v * xv.y;
                    acc[m][2] += v * xv.z;
                    acc[m][3] += v * xv.w;
                } else {
                    acc[m][0] += v * __ldg(xr + off);
                }
            }
        }
    }
    VT *yr = Y + row * k;
#pragma unroll
    for (int m = 0; m < NV; ++m) {
        const int off = (m * G + g) * VEC;
        if constexpr (VEC == 2) {
            __stcs(reinterpret_cast<double2 *>(yr + off), make_double2(acc[m][0], acc[m][1]));
        } else if constexpr (VEC == 4) {
            __stcs(reinterpret_cast<float4 *>(yr + off), make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]));
        } else {
            __stcs(yr + off, acc[m][0]);
        }
    }
}

template <int G> __device__ __forceinline__ unsigned group_mask(int lane) {
    return (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane - lane % G));
}

// a grid of all rows, one group of G lanes per row
template <typename VT, int G, int NV, int VEC>
__global__ void __launch_bounds__(256) spmm_row_major_kernel(const int *__restrict__ row_ptr,
                                                             const int *__restrict__ col,
                                                             const VT *__restrict__ val, int64_t n_rows, int64_t k,
                                                             const VT *__restrict__ X, VT *__restrict__ Y) {
    const int lane = threadIdx.x & 31;
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (row >= n_rows) return;  // whole groups leave together
    spmm_row<VT, G, NV, VEC>(row, lane % G, group_mask<G>(lane), row_ptr, col, val, k, X, Y);
}

// -------------------------------------------------------------- groups ----
// Warps of a CTA (one CTA per SM) and entries whose rows of X are loaded at a
// time, by the vectors a lane holds.  One vector: 24 warps of four entries (27-
// point 128^3, k = 16 FP64: 16 warps of eight took 713 us, 24 of four 569, both
// with rows taken from the counter).  More: 16 warps, which have the registers
// for it (lognormal, k = 48 FP64: 807 us against 957 with 24).
__host__ __device__ constexpr int group_warps(int nv) { return nv == 1 ? 24 : 16; }
__host__ __device__ constexpr int group_unroll(int nv) { return nv == 4 ? 2 : 4; }
constexpr int kStagePad = 4;  // entries between the staged rows: their 16-byte reads spread over the banks

// bytes of one stage of a warp: RW rows of CH + kStagePad values, then columns
template <typename VT> __host__ __device__ constexpr int stage_bytes(int rw, int ch) {
    return rw * (ch + kStagePad) * (int)(sizeof(VT) + sizeof(int));
}

// the most that the two stages of a CTA's warps take: launch_groups gives them 256 entries at most, or 32 rows of 4
template <typename VT> constexpr int stages_most(int warps) { return warps * 2 * stage_bytes<VT>(32, 8); }

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async4(unsigned dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// VB bytes of X as VB / sizeof(VT) values
template <typename VT, int VB> struct XVec {
    static constexpr int N = VB / (int)sizeof(VT);
    VT v[N];
    __device__ __forceinline__ void load(const VT *p) {
        if constexpr (VB == 16 && sizeof(VT) == 8) {
            const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
            v[0] = a.x; v[1] = a.y;
        } else if constexpr (VB == 16) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        } else if constexpr (VB == 8 && sizeof(VT) == 4) {
            const float2 a = __ldg(reinterpret_cast<const float2 *>(p));
            v[0] = a.x; v[1] = a.y;
        } else {
            v[0] = __ldg(p);
        }
    }
};

template <typename VT> __device__ __forceinline__ void read4(const VT *p, VT (&v)[4]) {
    if constexpr (sizeof(VT) == 8) {
        const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    }
}

// The sums of a column-major block: eight products at a time are summed plainly, and
// those sums in 64 bits for FP32; for FP64, with the rounding errors of the additions
// beside the sum.
template <typename VT> struct Plain {
    VT sum;
    __device__ __forceinline__ void add(VT x) { sum += x; }
};
struct Wide {
    double sum;
    __device__ __forceinline__ void add(float x) { sum += x; }
    __device__ __forceinline__ float value() const { return (float)sum; }
};
struct Compensated {
    double sum, err;
    __device__ __forceinline__ void add(double x) {
        const double s = sum + x, b = s - sum;
        err += (sum - (s - b)) + (x - b);
        sum = s;
    }
    // (infinities and NaN are the sum's: what stands beside them is no error)
    __device__ __forceinline__ double value() const { return isfinite(err) ? sum + err : sum; }
};

// U staged entries: their rows of X are all loaded before the first is used.
// AT: VT itself, or one of the sums above, which takes the U products together.
template <typename VT, typename AT, int VB, int NV, int U>
__device__ __forceinline__ void take(const int *sc, const VT *sv, const VT *const (&xl)[NV], int ldx,
                                     AT (&acc)[NV][XVec<VT, VB>::N]) {
    XVec<VT, VB> x[U][NV];
    int c[U];
    if constexpr (U % 4 == 0) {
#pragma unroll
        for (int u = 0; u < U; u += 4) {
            const int4 c4 = *reinterpret_cast<const int4 *>(sc + u);
            c[u] = c4.x; c[u + 1] = c4.y; c[u + 2] = c4.z; c[u + 3] = c4.w;
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = sc[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int m = 0; m < NV; ++m) x[u][m].load(xl[m] + (int64_t)c[u] * ldx);
    VT v[U];
    if constexpr (U % 4 == 0) {
#pragma unroll
        for (int u = 0; u < U; u += 4) {
            VT v4[4];
            read4<VT>(sv + u, v4);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[u + i] = v4[i];
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = sv[u];
    }
    if constexpr (std::is_same<VT, AT>::value) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < NV; ++m)
#pragma unroll
                for (int i = 0; i < XVec<VT, VB>::N; ++i) acc[m][i] += v[u] * x[u][m].v[i];
    } else {
#pragma unroll
        for (int m = 0; m < NV; ++m)
#pragma unroll
            for (int i = 0; i < XVec<VT, VB>::N; ++i) {
                VT sum = v[0] * x[0][m].v[i];
#pragma unroll
                for (int u = 1; u < U; ++u) sum += v[u] * x[u][m].v[i];
                acc[m][i].add(sum);
            }
    }
}

// Columns [0, kcols) of one panel: nvec vectors of a row of X (row stride ldx
// values).  COL: Y is column-major, element (row, v) at row + v * ldy, else
// row-major with row stride ldy.
// REG: no row has more than CH entries; rows are then dealt out in turn and a
// row is one chunk.  Otherwise the groups take rows from a shared counter, and
// leave out those of more than `limit` entries.
template <typename VT, int VB, int NV, bool COL, bool REG>
__global__ void __launch_bounds__(group_warps(NV) * 32, 1)
    spmm_group_kernel(const int *__restrict__ row_ptr, const int *__restrict__ col, const VT *__restrict__ val,
                      const int64_t *__restrict__ ranges, int G, int ch_shift, int nvec, int kcols, int ldx,
                      const VT *__restrict__ X, VT *__restrict__ Y, int64_t ldy, int limit) {
    using XV = XVec<VT, VB>;
    constexpr int VEC = XV::N;
    using AT = typename std::conditional<!COL, VT, typename std::conditional<sizeof(VT) == 8, Compensated, Wide>::type>::type;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int next_row;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int RW = 32 / G, CH = 1 << ch_shift;
    const int g = min(lane / G, RW - 1), gl = lane - g * G;  // lanes past the last group have gl >= G
    const int stage = stage_bytes<VT>(RW, CH);
    VT *sv0 = reinterpret_cast<VT *>(smem + (size_t)warp * 2 * stage) + g * (CH + kStagePad);
    int *sc0 = reinterpret_cast<int *>(smem + (size_t)warp * 2 * stage + RW * (CH + kStagePad) * sizeof(VT)) +
               g * (CH + kStagePad);
    const int r0 = (int)ranges[blockIdx.x], r1 = (int)ranges[blockIdx.x + 1];
    if constexpr (!REG) {
        if (threadIdx.x == 0) next_row = r0;
        __syncthreads();
    }
    const bool worker = gl < G;

    // the lane's vectors of a row; a lane without an m-th vector reads vector 0 and stores nothing
    const VT *xl[NV];
#pragma unroll
    for (int m = 0; m < NV; ++m) xl[m] = X + (worker && m * G + gl < nvec ? (m * G + gl) * VEC : 0);

    // the group's next row and its bounds (row >= r1: none left)
    auto grab = [&](bool need, int &row, int &s, int &e) {
        // one atomic per warp for the groups that need a row
        const unsigned want = __ballot_sync(0xffffffffu, need && gl == 0);
        if (!want) return;
        int base = 0;
        if (lane == 0) base = atomicAdd(&next_row, __popc(want));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (need) {
            row = base + __popc(want & ((1u << (g * G)) - 1u));
            s = e = 0;
            if (row < r1) {
                s = row_ptr[row];
                e = row_ptr[row + 1];
                if (COL && e - s > limit) {  // left out: e < s
                    s = 0;
                    e = -1;
                }
            }
        }
    };
    // entries [at, at + CH) of a row that ends at e into stage b
    auto issue = [&](int b, int at, int e) {
        VT *sv = reinterpret_cast<VT *>(reinterpret_cast<unsigned char *>(sv0) + b * stage);
        int *sc = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(sc0) + b * stage);
        if (worker)
            for (int j = gl; j < CH && j < e - at; j += G) {
                cp_async4(smem_u32(sc + j), col + at + j);
                if constexpr (sizeof(VT) == 8) cp_async8(smem_u32(sv + j), val + at + j);
                else cp_async4(smem_u32(sv + j), val + at + j);
            }
        cp_async_commit();
    };

    AT acc[NV][VEC];
#pragma unroll
    for (int m = 0; m < NV; ++m)
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[m][i] = AT{};

    // a plain sum of some entries to the row's
    using Part = Plain<VT>;
    auto fold = [&](const Part(&part)[NV][VEC]) {
        if constexpr (COL) {
#pragma unroll
            for (int m = 0; m < NV; ++m)
#pragma unroll
                for (int i = 0; i < VEC; ++i) acc[m][i].add(part[m][i].sum);
        }
    };
    // the entries of a staged chunk, n of them, into acc
    auto chunk = [&](int b, int n) {
        const VT *sv = reinterpret_cast<const VT *>(reinterpret_cast<unsigned char *>(sv0) + b * stage);
        const int *sc = reinterpret_cast<const int *>(reinterpret_cast<unsigned char *>(sc0) + b * stage);
        // U entries' vectors of X are loaded before any is used; with several vectors a
        // lane, fewer entries at a time, for the same bytes in flight
        constexpr int U = group_unroll(NV);
        int j = 0;
        if constexpr (COL) {
            for (; j + 2 * U <= n; j += 2 * U) {
                Part part[NV][VEC] = {};
                take<VT, Part, VB, NV, U>(sc + j, sv + j, xl, ldx, part);
                take<VT, Part, VB, NV, U>(sc + j + U, sv + j + U, xl, ldx, part);
                fold(part);
            }
            if (j < n) {
                Part part[NV][VEC] = {};
                if (j + U <= n) {
                    take<VT, Part, VB, NV, U>(sc + j, sv + j, xl, ldx, part);
                    j += U;
                }
                if constexpr (U > 2) {
                    if (j + 2 <= n) {
                        take<VT, Part, VB, NV, 2>(sc + j, sv + j, xl, ldx, part);
                        j += 2;
                    }
                }
                if (j < n) take<VT, Part, VB, NV, 1>(sc + j, sv + j, xl, ldx, part);
                fold(part);
            }
        } else {
            for (; j + U <= n; j += U) take<VT, AT, VB, NV, U>(sc + j, sv + j, xl, ldx, acc);
            if constexpr (U > 2) {
                if (j + 2 <= n) {
                    take<VT, AT, VB, NV, 2>(sc + j, sv + j, xl, ldx, acc);
                    j += 2;
                }
            }
            if (j < n) take<VT, AT, VB, NV, 1>(sc + j, sv + j, xl, ldx, acc);
        }
    };
    // the finished row to Y (store: it was not left out), and acc back to zero
    auto finish = [&](int row, bool store) {
#pragma unroll
        for (int m = 0; m < NV; ++m) {
            const int off = (m * G + gl) * VEC;
            if (worker && (!COL || store) && row < r1 && m * G + gl < nvec) {
                if constexpr (COL) {
#pragma unroll
                    for (int i = 0; i < VEC; ++i)
                        if (off + i < kcols) __stcs(Y + (int64_t)(off + i) * ldy + row, acc[m][i].value());
                } else {
                    VT *y = Y + (int64_t)row * ldy + off;
                    if constexpr (VB == 16 && sizeof(VT) == 8)
                        __stcs(reinterpret_cast<double2 *>(y), make_double2(acc[m][0], acc[m][1]));
                    else if constexpr (VB == 16)
                        __stcs(reinterpret_cast<float4 *>(y),
                               make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]));
                    else if constexpr (VB == 8 && sizeof(VT) == 4)
                        __stcs(reinterpret_cast<float2 *>(y), make_float2(acc[m][0], acc[m][1]));
                    else
                        __stcs(y, acc[m][0]);
                }
            }
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[m][i] = AT{};
        }
    };

    int row, s, e, row1, s1, e1, b = 0;
    if constexpr (REG) {
        const int stride = (int)(blockDim.x >> 5) * RW;
        auto bounds = [&](int r, int &s, int &e) {
            s = e = 0;
            if (r < r1) {
                s = row_ptr[r];
                e = row_ptr[r + 1];
            }
        };
        int wr = r0 + warp * RW;  // the warp's first row
        row = wr + g;
        bounds(row, s, e);
        issue(0, s, e);
        bounds(row + stride, s1, e1);
        for (; wr < r1; wr += stride, row += stride, b ^= 1) {
            issue(b ^ 1, s1, e1);
            int s2, e2;
            bounds(row + 2 * stride, s2, e2);
            cp_async_wait<1>();
            __syncwarp();
            chunk(b, e - s);
            __syncwarp();
            finish(row, true);
            s = s1;
            e = e1;
            s1 = s2;
            e1 = e2;
        }
    } else {
        // row: computed; row1: staged next; row2: its bounds are loaded
        int row2, s2, e2;
        grab(true, row, s, e);
        grab(true, row1, s1, e1);
        grab(true, row2, s2, e2);
        issue(0, s, e);
        while (__any_sync(0xffffffffu, row < r1)) {
            const bool more = e - s > CH;
            issue(b ^ 1, more ? s + CH : s1, more ? e : e1);
            cp_async_wait<1>();
            __syncwarp();
            chunk(b, min(e - s, CH));
            __syncwarp();
            if (more) {
                s += CH;
            } else {
                finish(row, e >= s);
                row = row1;
                s = s1;
                e = e1;
                row1 = row2;
                s1 = s2;
                e1 = e2;
            }
            grab(!more, row2, s2, e2);
            b ^= 1;
        }
    }
    cp_async_wait<0>();
}

// One warp per piece of a long row, for up to 32 vectors (a panel, blockIdx.y):
// a lane per vector and 32 / G entries side by side, four of them in flight a
// lane; then the lanes of one vector are added up.  part: kq sums a piece.
// Bound by the gathers of X, as the group kernel is.  10^6 rows of 5 entries, one
// of 10^6, k = 8 column-major FP64: 112 ms with that row left to a group, 0.19 ms now.
template <typename VT>
__global__ void __launch_bounds__(256) spmm_piece_kernel(const int2 *__restrict__ pieces, int64_t n_pieces,
                                                         const int *__restrict__ col, const VT *__restrict__ val,
                                                         int64_t nvec, int64_t ldx, const VT *__restrict__ X,
                                                         int64_t kq, double *__restrict__ part) {
    using XV = XVec<VT, 16>;
    constexpr int VEC = XV::N, U = 4;
    const int lane = threadIdx.x & 31;
    const int64_t p = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (p >= n_pieces) return;
    const int2 piece = pieces[p];
    const int64_t panels = (nvec + 31) / 32;
    for (int64_t pn = blockIdx.y; pn < panels; pn += gridDim.y) {
        const int64_t v0 = nvec * pn / panels;
        const int G = (int)(nvec * (pn + 1) / panels - v0), R = 32 / G;
        const int slot = lane / G, gl = lane - slot * G;
        const VT *xl = X + (v0 + gl) * VEC;
        double acc[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] = 0;
        if (slot < R) {
            // (left counts the entries: an entry's number plus a step may pass 2^31)
            int left = piece.y - piece.x - slot;
            const int *cp = col + piece.x + slot;
            const VT *vp = val + piece.x + slot;
            for (; left > 0; left -= U * R, cp += U * R, vp += U * R) {
                int c[U];
                VT v[U];
                XV x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool ok = u * R < left;
                    c[u] = ok ? ld_stream(cp + u * R) : -1;
                    v[u] = ok ? ld_stream(vp + u * R) : VT(0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (c[u] >= 0) x[u].load(xl + (int64_t)c[u] * ldx);
#pragma unroll
                for (int i = 0; i < VEC; ++i) {
                    VT sum = VT(0);
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (c[u] >= 0) sum += v[u] * x[u].v[i];
                    acc[i] += sum;
                }
            }
        }
        int o = 1;
        while (o < R) o <<= 1;
        for (o >>= 1; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                const double other = __shfl_down_sync(0xffffffffu, acc[i], o * G);
                if (slot < o && slot + o < R) acc[i] += other;
            }
        if (slot == 0)
#pragma unroll
            for (int i = 0; i < VEC; ++i) part[p * kq + (v0 + gl) * VEC + i] = acc[i];
    }
}

// The pieces of a long row (blockIdx.x), added up: W vectors side by side, 256 / W
// stretches of pieces, those in order.  long_rows: row, first piece, pieces.
template <typename VT>
__global__ void __launch_bounds__(256) spmm_combine_kernel(const int4 *__restrict__ long_rows,
                                                           const double *__restrict__ part, int64_t k, int64_t kq,
                                                           int W, VT *__restrict__ Y, int64_t ldy) {
    __shared__ Compensated sums[256];
    const int4 L = long_rows[blockIdx.x];
    const int t = threadIdx.x % W, stretch = threadIdx.x / W, S = 256 / W;
    const int p0 = (int)((int64_t)L.z * stretch / S), p1 = (int)((int64_t)L.z * (stretch + 1) / S);
    for (int64_t v0 = (int64_t)blockIdx.y * W; v0 < k; v0 += (int64_t)gridDim.y * W) {
        const int64_t v = v0 + t;
        Compensated s{0, 0};
        if (v < k) {
            const double *q = part + (int64_t)L.y * kq + v;
#pragma unroll 4
            for (int p = p0; p < p1; ++p) s.add(q[p * kq]);
        }
        sums[threadIdx.x] = s;
        __syncthreads();
        if (stretch == 0 && v < k) {
            for (int i = 1; i < S; ++i) {
                s.add(sums[i * W + t].sum);
                s.err += sums[i * W + t].err;
            }
            Y[v * ldy + L.x] = (VT)s.value();
        }
        __syncthreads();
    }
}

// weight[r]: a row's entries (none for one cut into pieces) and its Y write
__global__ void row_weights_kernel(const int *__restrict__ row_ptr, int64_t n, int limit, int64_t *__restrict__ weight) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int len = row_ptr[r + 1] - row_ptr[r];
    weight[r] = 1 + (len > limit ? 0 : len);
}

// The rows of more than `limit` entries (row, first piece, pieces) and their
// pieces, rows in any order.  next: rows << 40 | pieces taken so far (2^31 entries are
// less than 2^24 rows of more than 128).
__global__ void long_rows_kernel(const int *__restrict__ row_ptr, int64_t n, int limit, unsigned long long *next,
                                 int4 *__restrict__ long_rows, int2 *__restrict__ pieces) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int s = row_ptr[r], len = row_ptr[r + 1] - s;
    if (len <= limit) return;
    const int size = piece_size(len), m = (len - 1) / size + 1;
    const unsigned long long at = atomicAdd(next, (1ull << 40) | (unsigned long long)m);
    const int first = (int)(at & ((1ull << 40) - 1));
    long_rows[at >> 40] = make_int4((int)r, first, m, 0);
    for (int i = 0; i < m; ++i)
        pieces[first + i] = make_int2(s + i * size, i + 1 < m ? s + (i + 1) * size : s + len);
}

// ranges[b] = first row r with w[r] >= b * w[n] / grid, where w[r] is what the rows
// before r weigh: their entries and their Y writes, row_ptr[r] + r unless
// given (without the rows cut into pieces)
__global__ void row_ranges_kernel(const int *__restrict__ row_ptr, const int64_t *__restrict__ weights, int64_t n,
                                  int grid, int64_t *__restrict__ ranges) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > grid) return;
    auto w = [&](int64_t r) { return weights ? (r > 0 ? weights[r - 1] : 0) : (int64_t)row_ptr[r] + r; };
    const int64_t target = w(n) * b / grid;
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (w(mid) < target) lo = mid + 1;
        else hi = mid;
    }
    ranges[b] = b == grid ? n : lo;
}

// T (n x kp, row-major, kp >= k, zeros beyond column k) = X (column-major, leading dimension ld)
constexpr int kTrRows = 32;
template <typename VT>
__global__ void __launch_bounds__(256) to_row_major_kernel(const VT *__restrict__ X, int64_t n, int k, int kp,
                                                           int64_t ld, VT *__restrict__ T) {
    // 32 rows by up to 64 columns through shared memory: both sides coalesced
    __shared__ VT tile[64][kTrRows + 1];
    const int64_t r0 = (int64_t)blockIdx.x * kTrRows;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int v0 = blockIdx.y * 64; v0 < kp; v0 += gridDim.y * 64) {
        const int nv = min(64, kp - v0);
        for (int v = w; v < nv; v += 8)
            tile[v][lane] = (v0 + v < k && r0 + lane < n) ? ld_stream(X + (int64_t)(v0 + v) * ld + r0 + lane) : VT(0);
        __syncthreads();
        for (int i = threadIdx.x; i < kTrRows * nv; i += 256) {
            const int r = i / nv, v = i - r * nv;
            if (r0 + r < n) T[(r0 + r) * kp + v0 + v] = tile[v][r];
        }
        __syncthreads();
    }
}

template <typename VT, int G, int NV, int VEC>
void launch_rm(const DevCRS &a, int64_t k, const VT *X, VT *Y, cudaStream_t st) {
    const uint64_t threads = (uint64_t)a.n_rows * G;
    spmm_row_major_kernel<VT, G, NV, VEC><<<ceil_div_u(threads, 256), 256, 0, st>>>(a.rp(), a.ci(),
                                                                                    a.val.template as<VT>(),
                                                                                    a.n_rows, k, X, Y);
}

// Lanes per row and vectors per lane for a panel of nvec vectors: the pair
// that keeps most lanes busy, with at least four rows a warp where it can.
void group_shape(int nvec, int &G, int &NV) {
    double best = 0;
    for (int nv : {1, 2, 4}) {
        const int gg = (nvec + nv - 1) / nv;
        if (gg > 32) continue;
        double score = (double)nvec * (32 / gg) / (32.0 * nv);
        if (gg > 8) score *= 0.8;
        score *= nv == 1 ? 1.0 : (nv == 2 ? 0.99 : 0.97);
        if (score > best) {
            best = score;
            G = gg;
            NV = nv;
        }
    }
}

// the long rows of a column-major Y; X: rows of ldx values, whole vectors
template <typename VT>
void launch_pieces(const DevCRS &a, const SpmmPlan &p, int64_t k, int64_t ldx, const VT *X, VT *Y, int64_t ldy,
                   cudaStream_t st) {
    const int64_t nvec = ldx / V16<VT>::N;
    const unsigned panels = (unsigned)std::min<int64_t>((nvec + 31) / 32, 65535);
    spmm_piece_kernel<VT><<<dim3(ceil_div_u(p.n_pieces, 8), panels), 256, 0, st>>>(
        p.pieces.as<int2>(), p.n_pieces, a.ci(), a.val.template as<VT>(), nvec, ldx, X, ldx, p.part.as<double>());
    SMAX_CUDA(cudaGetLastError());
    int W = 1;
    while (W < 32 && W < k) W <<= 1;
    const dim3 grid(p.n_long, (unsigned)std::min<int64_t>((k + W - 1) / W, 65535));
    spmm_combine_kernel<VT><<<grid, 256, 0, st>>>(p.long_rows.as<int4>(), p.part.as<double>(), k, ldx, W, Y, ldy);
    SMAX_CUDA(cudaGetLastError());
}

template <typename VT, int VB, bool COL>
void launch_groups(const DevCRS &a, const SpmmPlan &p, int64_t k, int64_t ldx, const VT *X, VT *Y, int64_t ldy,
                   cudaStream_t st) {
    constexpr int VEC = VB / (int)sizeof(VT);
    const int64_t nvec_all = (k + VEC - 1) / VEC;
    const int64_t panels = (nvec_all + 127) / 128;
    for (int64_t pn = 0; pn < panels; ++pn) {
        const int64_t v0 = nvec_all * pn / panels, v1 = nvec_all * (pn + 1) / panels;
        const int nvec = (int)(v1 - v0);
        const int kcols = (int)std::min<int64_t>(k - v0 * VEC, (int64_t)nvec * VEC);
        int G = 1, NV = 1;
        group_shape(nvec, G, NV);
        const int rw = 32 / G;
        // a chunk holds a row of mean length, and of far longer rows, which are a
        // chain of chunks, a sixteenth; a warp's stage at most 256 entries (rows of 1
        // entry, one in 1000 of 500, 20000 rows, k = 3 FP32: 88 us with chunks of 4, 56
        // with 16; lognormal 600000 rows, k = 20 FP32: 195 with 16, 182 with 32)
        int shift = 2;
        while (shift < 5 && (rw << (shift + 1)) <= 256 &&
               ((int64_t)a.n_rows << shift < a.nnz || p.longest > 16 << shift))
            ++shift;
        // rows of nearly equal length: a chunk that holds the longest
        bool reg = false;
        if (p.regular) {
            int sh = shift;
            while (sh < 5 && (1 << sh) < p.longest && (rw << (sh + 1)) <= 256) ++sh;
            reg = (1 << sh) >= p.longest;
            if (reg) shift = sh;
        }
        auto go = [&](auto kern, int warps) {
            const size_t sm = (size_t)warps * 2 * stage_bytes<VT>(rw, 1 << shift);
            // set on every call: the attribute belongs to the current device; always to the most
            // that a call can need: it is one for all threads, and another's launch
            // may come between this and the launch below
            SMAX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, stages_most<VT>(warps)));
            kern<<<p.grid, warps * 32, sm, st>>>(a.rp(), a.ci(), a.val.template as<VT>(), p.ranges.as<int64_t>(), G,
                                                 shift, nvec, kcols, (int)ldx, X + v0 * VEC,
                                                 COL ? Y + v0 * VEC * ldy : Y + v0 * VEC, ldy,
                                                 p.limit);
            SMAX_CUDA(cudaGetLastError());
        };
        auto pick = [&](auto NVc) {
            constexpr int N = NVc.value;
            if (reg) go(spmm_group_kernel<VT, VB, N, COL, true>, group_warps(N));
            else go(spmm_group_kernel<VT, VB, N, COL, false>, group_warps(N));
        };
        if (NV == 1) pick(std::integral_constant<int, 1>());
        else if (NV == 2) pick(std::integral_constant<int, 2>());
        else pick(std::integral_constant<int, 4>());
    }
}

// scalar fallback for any k: one warp per row, lanes over the k columns
template <typename VT>
__global__ void spmm_row_major_generic(const int *__restrict__ row_ptr, const int *__restrict__ col,
                                       const VT *__restrict__ val, int64_t n_rows, int64_t k,
                                       const VT *__restrict__ X, VT *__restrict__ Y) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= n_rows) return;
    const int s = row_ptr[row], e = row_ptr[row + 1];
    for (int64_t v = lane; v < k; v += 32) {
        VT acc = VT(0);
        for (int j = s; j < e; ++j) acc += val[j] * X[(int64_t)col[j] * k + v];
        Y[row * k + v] = acc;
    }
}

}  // namespace

// found[0]: entries of the longest row, [1]: rows of more than `limit`, [2]: their pieces
static __global__ void longest_row_kernel(const int *__restrict__ row_ptr, int64_t n, int limit,
                                          int *__restrict__ found) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int len = r < n ? row_ptr[r + 1] - row_ptr[r] : 0;
    if (len > limit) {
        atomicAdd(found + 1, 1);
        atomicAdd(found + 2, (len - 1) / piece_size(len) + 1);
    }
    len = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);
    if ((threadIdx.x & 31) == 0 && len > 0) atomicMax(found, len);
}

void SpmmPlan::build(const DevCRS &a, bool col_major, cudaStream_t st) {
    const int64_t n = a.n_rows;
    // cut: rows of more than a piece and four times the average
    limit = !col_major ? INT_MAX : (int)std::min<int64_t>(INT_MAX, std::max<int64_t>(kPiece, n > 0 ? 4 * a.nnz / n : 0));
    DevBuf d(sizeof(int) * 3);
    int h[3] = {0, 0, 0};
    SMAX_CUDA(cudaMemsetAsync(d.p, 0, sizeof(h), st));
    if (n > 0) longest_row_kernel<<<ceil_div_u(n, 256), 256, 0, st>>>(a.rp(), n, limit, d.as<int>());
    SMAX_CUDA(cudaMemcpyAsync(h, d.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    SMAX_CUDA(cudaStreamSynchronize(st));
    longest = h[0];
    n_long = h[1];
    n_pieces = h[2];
    regular = (int64_t)longest * n <= 2 * a.nnz + 8 * n;
    DevBuf weights, tmp, next;
    if (n_long > 0) {
        long_rows.ensure(sizeof(int4) * n_long);
        pieces.ensure(sizeof(int2) * n_pieces);
        next.alloc(sizeof(unsigned long long));
        SMAX_CUDA(cudaMemsetAsync(next.p, 0, sizeof(unsigned long long), st));
        long_rows_kernel<<<ceil_div_u(n, 256), 256, 0, st>>>(a.rp(), n, limit, next.as<unsigned long long>(),
                                                             long_rows.as<int4>(), pieces.as<int2>());
        weights.alloc(sizeof(int64_t) * n);
        int64_t *w = weights.as<int64_t>();
        row_weights_kernel<<<ceil_div_u(n, 256), 256, 0, st>>>(a.rp(), n, limit, w);
        SMAX_CUDA(cudaGetLastError());
        size_t tb = 0;
        SMAX_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tb, w, w, n, st));
        tmp.alloc(tb ? tb : 1);
        SMAX_CUDA(cub::DeviceScan::InclusiveSum(tmp.p, tb, w, w, n, st));
    }
    grid = sm_count();
    ranges.ensure(sizeof(int64_t) * (grid + 1));
    row_ranges_kernel<<<ceil_div_u((uint64_t)grid + 1, 256), 256, 0, st>>>(a.rp(), weights.as<int64_t>(), n, grid,
                                                                           ranges.as<int64_t>());
    SMAX_CUDA(cudaGetLastError());
    if (n_long > 0) SMAX_CUDA(cudaStreamSynchronize(st));  // the temporaries die here
}

// Whether a row-major product runs on the grid of all rows.  Rows of nearly
// equal length, a power of two of 16-byte vectors, and either a wide block,
// whose rows of X are more than an SM keeps (27-point 96^3, grid against
// groups: k = 64 FP64 655 / 801 us, k = 64 FP32 359 / 396, k = 128 FP64 1199 /
// 1997; k = 16 FP64 276 / 257), or rows too short to pay for the groups' work
// per row (7-point 100^3: k = 16 FP64 134 / 154 us, k = 16 FP32 79 / 83; k = 4
// FP64 73 / 48), or rows of X of one 16-byte FP64 vector (27-point 96^3, k = 2:
// 239 / 495 us).  Rows of uneven length take the groups (lognormal 500000,
// k = 64 FP64: 946 against 1543 us), except (grid / groups, us):
//  * one FP64 vector, if no row is long (2^17 rows of 2, one in 100 of 32: 18 / 23;
//    2^19 of 8, one in 100 of 64: 55 / 69; but of 3, one in 1000 of 100: 40 / 37) or if
//    there are many that are not short (lognormal 600000: 300 / 370; 150000: 131 / 109;
//    2^19 of 10, one in 1000 of 3000: 600 / 528);
//  * rows of fewer than four entries on average and none long, where the groups'
//    work per row and a CTA's start count: small matrices whatever the width (20000
//    rows, nine in ten empty, k = 32 FP64 16 / 26, k = 5 FP32 14 / 20; of 2 entries, one in
//    100 of 32, k = 20 FP32 14 / 16), wide blocks up to 2^18 rows, and beyond if few
//    rows are longer than the rest (2^19 of 2, one in 100 of 32, k = 32 FP64 115 / 122;
//    nine in ten empty 190 / 160); of fewer than 2.5 also narrow ones (2^17 of 2, one in
//    100 of 32, k = 8 FP64 20 / 24, FP32 20 / 22; 2^19: 40 / 40, 35 / 33).
// nvec: 16-byte vectors of a row of X, 0 if it is not whole vectors (the grid's
// kernel for such rows is a warp each).
static bool grid_suits(const DevCRS &a, const SpmmPlan &p, int64_t nvec, int vbytes) {
    const int64_t n = a.n_rows;
    const bool short_rows = a.nnz < 4 * n && p.longest <= 64;
    if (nvec <= 0 || nvec > 128 || (nvec & (nvec - 1))) return short_rows && n < (1 << 16);
    if (nvec == 1 && vbytes == 8) return p.regular || p.longest <= 64 || (n >= (1 << 18) && a.nnz >= 15 * n);
    if (nvec >= 8 && short_rows && (n < (1 << 18) || p.longest * n > 12 * a.nnz)) return true;
    if (short_rows && 2 * a.nnz < 5 * n && n >= (1 << 16) && n < (1 << 18)) return true;
    if (!p.regular) return false;
    return nvec >= 16 || (nvec >= 4 && a.nnz <= 12 * a.n_rows);
}

template <typename VT>
void crs_spmm_row_major(const DevCRS &a, int64_t k, const VT *X, VT *Y, cudaStream_t st, const SpmmPlan &plan,
                        int variant) {
    if (a.n_rows == 0 || k == 0) return;
    constexpr int VEC = V16<VT>::N;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y) | (k * sizeof(VT));
    const bool grid = variant == 1 || (variant == 0 && grid_suits(a, plan, (bits & 15) == 0 ? k / VEC : 0, sizeof(VT)));
    if (!grid && k > 1 && k < (1 << 30) && !near_int_end(a.n_rows)) {
        if ((bits & 15) == 0) launch_groups<VT, 16, false>(a, plan, k, k, X, Y, k, st);
        else if ((bits & 7) == 0 || sizeof(VT) == 8) launch_groups<VT, 8, false>(a, plan, k, k, X, Y, k, st);
        else launch_groups<VT, sizeof(VT), false>(a, plan, k, k, X, Y, k, st);
        return;
    }
    const int64_t nvec = (bits & 15) == 0 ? k / VEC : 0;
    bool done = true;
    switch (nvec) {
    case 1: launch_rm<VT, 1, 1, VEC>(a, k, X, Y, st); break;
    case 2: launch_rm<VT, 2, 1, VEC>(a, k, X, Y, st); break;
    case 4: launch_rm<VT, 4, 1, VEC>(a, k, X, Y, st); break;
    case 8: launch_rm<VT, 8, 1, VEC>(a, k, X, Y, st); break;
    case 16: launch_rm<VT, 8, 2, VEC>(a, k, X, Y, st); break;
    case 32: launch_rm<VT, 8, 4, VEC>(a, k, X, Y, st); break;
    case 64: launch_rm<VT, 16, 4, VEC>(a, k, X, Y, st); break;
    case 128: launch_rm<VT, 32, 4, VEC>(a, k, X, Y, st); break;
    default: done = false;
    }
    if (!done) {
        if (k == 1) launch_rm<VT, 1, 1, 1>(a, k, X, Y, st);
        else
            spmm_row_major_generic<VT><<<ceil_div_u((uint64_t)a.n_rows * 32, 256), 256, 0, st>>>(
                a.rp(), a.ci(), a.val.template as<VT>(), a.n_rows, k, X, Y);
    }
    SMAX_CUDA(cudaGetLastError());
}

// Whether a column-major block runs as one product per column: rows so short
// that transposing X costs more than reading A again.  2^19 rows of 2 entries,
// one in 100 of 32, FP64: k = 3 37 us as products, 52 as a block; k = 8 89 and
// 70; below 2^17 rows the products' launches cost more (20000 rows, k = 3: 27
// and 21).  With rows of more than 64 times the average length also k = 8 (of 1
// entry, one in 1000 of 500: 137 and 173 us).  Of longer rows, two vectors
// where their lengths differ (products and block, lognormal 30000 rows FP64 28 and 47 us, 300000
// 66 and 141; 2^19 rows of 8, one in 100 of 64: 60 and 89; 20000 of these 27 and
// 23) and three where some are far longer (lognormal 30000 FP32 37 and 47, 300000 92 and 105).
// Two vectors of even rows too, once A is large: a lane then has a row to itself and
// waits for a vector of X per entry.  27-point 24^3 FP64 19 and 20, 40^3 26 and 38, 96^3
// 166 and 532; FP32 40^3 22 and 23, 64^3 43 and 61, 96^3 106 and 159; 40000 rows of 100
// FP32 66 and 50, 200000 179 and 257.  Rows of hundreds keep their lanes waiting for
// the longest already where it has a quarter more than the average (3000 rows of 50 to
// 150 FP64 30 and 38, 1500 of 100 to 300 35 and 50; three vectors, 1111 of 450 to 1350
// 83 and 108; 1500 of 200 each 35 and 34).  And, of many short rows, where the copies of X
// and the columns of Y outweigh A: three vectors (7-point 200^3 FP64 522 and 637, FP32
// 351 and 476; 3.3 million rows of 6 FP64 301 and 346), in FP32 of rows below 8 entries
// also four to six (7-point 200^3 447 and 487, 557 and 682, 658 and 688; 13 million
// rows of 6, k = 6 1952 and 2439).
bool spmm_by_columns(const DevCRS &a, int64_t k, int vbytes, int64_t longest) {
    if (near_int_end(a.n_rows) || k >= (1 << 30)) return true;
    const bool skewed = longest * a.n_rows > 64 * a.nnz;
    const bool uneven = longest * a.n_rows > 2 * a.nnz + 8 * a.n_rows;
    if (a.nnz < 4 * a.n_rows) return (k < 8 && a.n_rows >= (1 << 17)) || (k <= 8 && skewed);
    if (k == 2 && a.nnz >= (vbytes == 8 ? 1 << 19 : a.nnz < 64 * a.n_rows ? 1 << 21 : 1 << 23)) return true;
    if (k == 3 && a.n_rows >= (1 << 21) && a.nnz < 16 * a.n_rows) return true;
    if (k <= 6 && vbytes == 4 && a.n_rows >= (1 << 22) && a.nnz < 8 * a.n_rows) return true;
    const bool long_uneven = a.nnz >= (k == 2 ? 64 : 512) * a.n_rows && 4 * longest * a.n_rows > 5 * a.nnz;
    if (k <= 3 && a.nnz >= (1 << 18) && long_uneven) return true;
    return a.nnz >= (1 << 18) && ((k == 2 && uneven) || (k == 3 && longest * a.n_rows > 32 * a.nnz));
}

int64_t spmm_col_major_work(int64_t n_cols, int64_t k, int vbytes) {
    const int64_t per = 16 / vbytes, kp = (k + per - 1) / per * per;
    return n_cols * kp * vbytes;
}

template <typename VT>
void crs_spmm_col_major(const DevCRS &a, int64_t k, const VT *X, VT *Y, int64_t ld, VT *work, cudaStream_t st,
                        const SpmmPlan &plan) {
    if (a.n_rows == 0 || k == 0) return;
    constexpr int VEC = V16<VT>::N;
    const int64_t kp = (k + VEC - 1) / VEC * VEC;
    to_row_major_kernel<VT><<<dim3(ceil_div_u(a.n_cols, kTrRows), std::min(ceil_div_u(kp, 64), 65535u)), 256, 0, st>>>(
        X, a.n_cols, (int)k, (int)kp, ld, work);
    SMAX_CUDA(cudaGetLastError());
    if (plan.n_long > 0) launch_pieces<VT>(a, plan, k, kp, work, Y, ld, st);
    launch_groups<VT, 16, true>(a, plan, k, kp, work, Y, ld, st);
}

template void crs_spmm_col_major<double>(const DevCRS &, int64_t, const double *, double *, int64_t, double *,
                                         cudaStream_t, const SpmmPlan &);
template void crs_spmm_col_major<float>(const DevCRS &, int64_t, const float *, float *, int64_t, float *,
                                        cudaStream_t, const SpmmPlan &);
template void crs_spmm_row_major<double>(const DevCRS &, int64_t, const double *, double *, cudaStream_t,
                                         const SpmmPlan &, int);
template void crs_spmm_row_major<float>(const DevCRS &, int64_t, const float *, float *, cudaStream_t,
                                        const SpmmPlan &, int);

}  // namespace smax
