// sweep.cuh -- triangular solves swept level by level on one CTA per
// right-hand side (sweep.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace smax {

// Rows in sweep order ("positions").  A run of narrow levels is swept by one
// CTA that keeps the last kRing solutions in shared memory; everything else it
// reads -- values, source codes, 1/diagonal and right-hand side -- is streamed
// into a shared-memory stage by bulk copies, several levels ahead.
//
// A level is one or more chunks of rows.  A chunk in the blob is a 48-byte
// header followed by the operands of its mp rows (the rows rounded up to a
// multiple of 4, so every block is 16-byte aligned): off-diagonal values,
// 1 / diagonal (or the diagonal itself: div) and a source code per entry:
// code >= 0 is a byte offset into the ring (a slot that holds 0, for padding),
// code < 0 the position ~code of x.  Rows of up to three entries are stored as
// 16-byte elements, wider ones as dense column-major blocks.
// Consecutive chunks form a record, the unit of one bulk copy (plus one for
// its right-hand sides).  Where each record lies in the stage and which
// records must be finished before it may be copied is fixed when the pack is
// built.  A level too wide for one CTA is a chunk of its own, read by a grid.
struct SweepPack {
    static constexpr int kRing = 8192;  // solutions kept in shared memory (positions; a power of 2)

    struct Wide {
        int pos, m, w, mp, off;  // first position, rows, width, padded rows, blob offset / 16
    };
    static constexpr int kGroups = 4;  // groups of threads that take a run's chunks in turn
    struct Run {
        int rec0, n_rec;  // records
        int pos0, pos1;   // positions [pos0, pos1)
        int n_levels;
        int level_chunks;               // arrivals of a level, in chunks: the most a level has
        int at[kGroups], rec[kGroups];  // stage offset (-1: none) and record of each group's first chunk
    };
    struct Item {
        bool wide;
        int index;    // into wides or runs
        int threads;  // of a group of a run's CTA
    };
    int64_t n = 0, npos = 0;
    int n_chunks = 0;
    int vbytes = 8;
    bool div = false;
    int stage_bytes = 0;
    bool shared_sm = false;  // a batch whose CTAs share an SM by twos
    std::vector<Wide> wides;
    std::vector<Run> runs;
    std::vector<Item> items;
    int64_t blob_bytes = 0;
    DevBuf prow;    // int[npos]: row of each position, -1 for padding
    DevBuf pchunk;  // int[npos]: chunk of each position
    DevBuf chunks;  // ChunkDesc[n_chunks] (sweep.cu)
    DevBuf blob, recs, drun;
    DevBuf bp, xp;  // VT[vectors][npos]: right-hand sides and solutions in position order
    int vectors = 0;  // right-hand sides solved at a time
    int most_vectors = 1 << 30;  // as many as there was memory for
    bool needs_x_init = false;  // some entry reads a solution not computed before it
};

// How long the waits of a sweep last.
struct SweepWait {
    static constexpr long long kPollNs = 128;  // a limit given in polls counts this many nanoseconds for each
    long long ns = 20000000 * kPollNs;
    bool never = false;  // test: the levels wait for an arrival that never comes
    bool operator!=(const SweepWait &o) const { return ns != o.ns || never != o.never; }
};

struct SweepStep {
    int first, count, kind;  // first sweep step, steps, kind 0: a wide level (grid) / 1: a run (one CTA)
};

// Builds the pack of a triangular CRS matrix (diagonal last in each row, D its
// diagonal) whose sweep step s solves the rows order[src_begin[s] ..
// src_begin[s] + count[s]) (order == nullptr: the identity); `steps` groups the
// sweep steps.  div: divide by the diagonal instead of multiplying by its
// reciprocal.  batch: the runs are independent matrices (sweep_solve_batch).  Returns false when the
// padding would make the pack more than about three times the off-diagonal
// entries, or a level takes so long that others' waits for it could give up, or
// has more chunks than an mbarrier counts arrivals.
// Synchronises.
bool build_sweep_pack(SweepPack &pk, const int *rp, const int *ci, const void *val, const void *D, int vbytes,
                      int64_t n, const int *order, const std::vector<int> &src_begin, const std::vector<int> &count,
                      const std::vector<SweepStep> &steps, bool div, bool batch, cudaStream_t st);

// New values (and diagonal) of the matrix the pack was built from.
void refill_sweep_pack(SweepPack &pk, const int *rp, const void *val, const void *D, cudaStream_t st);

// Workspace for solves of up to k right-hand sides (allocates: call outside
// stream capture).  Solves take as many at a time as it holds: half as many, and
// so on, if there is no memory for k.
void sweep_reserve(SweepPack &pk, int64_t k);

// Solves k right-hand sides, element (r, v) of B and X at r * rs + v * vs.
// status (may be null) gets SMAX_ERR_TIMEOUT if a wait gives up; the solutions
// of its run are then NaN.
template <typename VT>
void sweep_solve(const SweepPack &pk, const VT *B, VT *X, int64_t k, int64_t rs, int64_t vs, DevStatus *status,
                 const SweepWait &wait, cudaStream_t st);

// One CTA per run, runs (independent matrices) taken from a device work queue
// in the order queue_order.  *status (which the host can read) becomes
// SMAX_ERR_TIMEOUT if a wait gives up; the solutions of that matrix and of those
// its CTA takes after it are then NaN.
template <typename VT>
void sweep_solve_batch(const SweepPack &pk, const int *queue_order, int n_mats, int *queue, const VT *B, VT *X,
                       int *status, const SweepWait &wait, cudaStream_t st);

}  // namespace smax
