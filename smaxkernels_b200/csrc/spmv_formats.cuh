// spmv_formats.cuh -- device-resident SELL-C-sigma and BCRS matrices, their
// SpMV launchers and the GPU conversions from CRS; SpMM launchers.
#pragma once

#include "common.cuh"

namespace smax {

// Device copy of a CRS matrix (int32 indices); col/val may be padded.
struct DevCRS {
    int64_t n_rows = 0, n_cols = 0, nnz = 0;
    DevBuf row_ptr, col, val;
    const int *rp() const { return row_ptr.as<int>(); }
    const int *ci() const { return col.as<int>(); }
};

// SELL-C-sigma (src/common.hpp:62-88)
struct DevSCS {
    int64_t C = 0, sigma = 0, n_rows = 0, n_rows_padded = 0, n_cols = 0, n_chunks = 0, n_elements = 0, nnz = 0;
    DevBuf chunk_ptr, chunk_len, col, val;
    // warp tasks of at most kScsTaskCols chunk columns (scs_plan): a chunk
    // longer than that is split, its tasks write partial sums to slots that a
    // fix-up pass adds in task order
    int64_t n_tasks = 0, n_multi = 0, n_slots = 0;
    DevBuf task_chunk, task_j0, task_slot, multi_chunk, multi_first, multi_count, partial;
    // per padded row: its entries up to the last one that is not padding
    // (column 0, value 0); the task kernel skips the rest when x[0] is finite
    DevBuf row_len;
    int plan_vbytes = 0;
};

constexpr int kScsTaskCols = 64;
// Builds the task plan of a SELL-C-sigma matrix (after upload or conversion).
void scs_plan(DevSCS &m, int vbytes, cudaStream_t st);

// BCRS (src/common.hpp:90-111): n_rows/n_cols count blocks
struct DevBCRS {
    int64_t n_rows = 0, n_cols = 0, n_blocks = 0, bh = 0, bw = 0, hpad = 0, wpad = 0;
    bool col_major = false;
    DevBuf row_ptr, col, val;
    // block rows longest first (bcrs_plan): the warp-per-block-row kernel
    // starts the long rows first, so none is left running alone at the end
    DevBuf order;
};
void bcrs_plan(DevBCRS &m, cudaStream_t st);

void validate_scs(const DevSCS &m, DevStatus *st, cudaStream_t s);
void validate_bcrs(const DevBCRS &m, DevStatus *st, cudaStream_t s);

template <typename VT> void scs_spmv(const DevSCS &m, const VT *x, VT *y, cudaStream_t st);
bool scs_vector_path(int64_t C, int vbytes);
// perm (device, n_rows ints) receives perm[old] = new
void crs_to_scs(const DevCRS &a, int vbytes, int64_t C, int64_t sigma, DevSCS &out, DevBuf &perm, cudaStream_t st);

template <typename VT> void bcrs_spmv(const DevBCRS &m, const VT *x, VT *y, cudaStream_t st);
// max_blocks >= 0: when the matrix needs more blocks, only out.n_blocks is set
// (out.val stays empty)
void crs_to_bcrs(const DevCRS &a, int vbytes, int64_t bh, int64_t bw, int64_t hpad, int64_t wpad, bool col_major,
                 DevBCRS &out, cudaStream_t st, int64_t max_blocks = -1);

// Y = A X with k right-hand sides.  Row-major: X[col*k+v], Y[row*k+v].
// Column-major: X[ldx*v+col], Y[row+ldy*v] (the reference uses A's n_rows as
// the leading dimension of X and Y, src/kernels/spmm/spmm_cpu/spmm_cpu_crs_impl.hpp:29,44).
// Row ranges of the SpMM kernel's CTAs: contiguous, each with its share of the nonzeros and rows.
struct SpmmPlan {
    DevBuf ranges;  // int64 row bounds, grid + 1 entries
    int grid = 0;
    int longest = 0;       // entries of the longest row
    bool regular = false;  // ... at most twice the mean plus 8
    // column-major blocks: rows of more than `limit` entries, cut into pieces (spmm.cu)
    int limit = 0, n_long = 0;
    int64_t n_pieces = 0;
    DevBuf long_rows;  // int4[n_long]: row, first piece, pieces
    DevBuf pieces;     // int2[n_pieces]: entries [x, y)
    DevBuf part;       // double[n_pieces][k rounded up]: their sums
    DevBuf work;    // column-major blocks: X as a row-major block
    int64_t part_bytes(int64_t k) const { return n_pieces * ((k + 3) / 4 * 4) * (int64_t)sizeof(double); }
    void build(const DevCRS &a, bool col_major, cudaStream_t st);
};
// variant 0: chosen by the matrix and the block's width; 1: a grid of all
// rows; 2: lane groups going through a range of rows per SM
template <typename VT>
void crs_spmm_row_major(const DevCRS &a, int64_t k, const VT *X, VT *Y, cudaStream_t st, const SpmmPlan &plan,
                        int variant = 0);
// whether a column-major block of k vectors runs as k products instead
bool spmm_by_columns(const DevCRS &a, int64_t k, int vbytes, int64_t longest);
// bytes of workspace crs_spmm_col_major needs for k vectors
int64_t spmm_col_major_work(int64_t n_cols, int64_t k, int vbytes);
template <typename VT>
void crs_spmm_col_major(const DevCRS &a, int64_t k, const VT *X, VT *Y, int64_t ld, VT *work, cudaStream_t st,
                        const SpmmPlan &plan);

}  // namespace smax
