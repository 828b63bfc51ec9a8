// levelpack.cuh -- level-ordered packed triangular matrices and the sync-free
// solves over them (levelpack.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace smax {

// Rows in sweep order ("positions") for the sync-free solves, each level stored
// as a dense column-major block of its rows' off-diagonal entries (ELL per
// level): the i-th entry of the t-th row of a level with m rows sits at
// base + i*m + t, so a warp reads its rows' i-th entries with one coalesced
// load.  An entry names its source row in the caller's numbering, or kPad.
// `tasks` lists the warp tasks in sweep order, up to 32 rows of one level
// each, so a warp's rows never depend on one another.
struct LevelPack {
    static constexpr int kPad = -0x7fffffff - 1;

    struct Level {
        int pos, m, w;      // first position, rows, width (max off-diagonals)
        int base;           // first entry (packs are limited to 2^31 entries)
    };
    int64_t n = 0, ents = 0;
    int vbytes = 8;
    int levels = 0;
    DevBuf prow;    // int[n]: row of each position
    DevBuf psrc;    // int[ents]
    DevBuf pval;    // VT[ents]
    DevBuf pinv;    // VT[n]: 1 / diagonal
    bool reads_unsolved = false;  // some entry reads a solution not computed before it
    DevBuf tasks;  // int4[n_tasks]: first position, rows | width << 6, level rows, first entry
    int n_tasks = 0;
    int n_levels() const { return levels; }
};

// Builds the pack of a triangular CRS matrix (diagonal last in each row, D its
// diagonal) for a sweep whose step s solves the rows order[src_begin[s] ..
// src_begin[s] + count[s]) (order == nullptr: the identity).  Returns false
// (building nothing) when the per-level padding would make the pack more than
// about three times the off-diagonal entries.  Synchronises.
bool build_level_pack(LevelPack &pk, const int *rp, const int *ci, const void *val, const void *D, int vbytes,
                      int64_t n, const int *order, const std::vector<int> &src_begin, const std::vector<int> &count,
                      cudaStream_t st);

// New values (and diagonal) of the matrix the pack was built from.
void refill_level_pack(LevelPack &pk, const int *rp, const void *val, const void *D, cudaStream_t st);

// Sync-free solve on the pack: X is first filled with a pending
// marker (a signalling-NaN pattern that no arithmetic result has), then one
// launch of warps takes 32-row tasks in sweep order (a CTA claims a chunk of
// tasks with one atomic) and each row waits on its sources' values in X,
// with no barrier between levels.  A row's sources lie in earlier tasks, which
// were claimed by running CTAs, so the earliest unfinished task can always
// finish.  Each wait gives up after `limit` polls: SMAX_ERR_TIMEOUT in st, an
// abort flag that ends the other waits, and NaN for the missing value.
// B and X must not overlap.  ctl: device scratch of at least 64 bytes.
// force_timeout (test only): the first row also waits on a word nothing writes.
template <typename VT>
void pack_solve_syncfree(const LevelPack &pk, const VT *B, VT *X, void *ctl, long long limit, bool force_timeout,
                         DevStatus *st, cudaStream_t s);

// The sync-free solve for k > 1 right-hand sides, on the matrix's own CRS
// arrays (diagonal last in each row) with the rows in the sweep order of a
// pack: a warp per row, lanes over vectors, bounded waits as
// above.  Blocks are row-major (r*k + v) or column-major (r + v*n, the
// matrix's row count as the leading dimension).  B and X (n * k values each)
// must not overlap.
template <typename VT>
void solve_syncfree_rows(const LevelPack &pk, const int *rp, const int *ci, const VT *val, const VT *D, const VT *B,
                         VT *X, int64_t k, bool row_major, void *ctl, long long limit, DevStatus *st, cudaStream_t s);

}  // namespace smax
