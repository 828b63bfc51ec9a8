// download.cuh -- large device-to-host copies into fresh pageable memory
// (download.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace smax {

struct DownloadPart {
    void *dst;
    const void *src;
    size_t bytes;
};

// Pinned staging of the downloads of one kernel object: allocated by the first
// large one, freed with the object.
struct DownloadStage {
    static constexpr int kWorkers = 6;           // host threads, two pieces each
    static constexpr size_t kPiece = 1u << 20;   // bytes of a piece
    static constexpr size_t kLarge = 4u << 20;   // smaller downloads are plain copies
    void *pinned = nullptr;
    cudaStream_t streams[kWorkers] = {};
    cudaEvent_t done[kWorkers][2] = {}, start = nullptr;
    bool ready = false, unfit = false;
    bool ensure();
    void release();
    DownloadStage() = default;
    DownloadStage(const DownloadStage &) = delete;
    DownloadStage &operator=(const DownloadStage &) = delete;
    ~DownloadStage() { release(); }
};

// Copies the parts, ordered after the work queued on st; returns when they are complete.
void download(DownloadStage &stage, const std::vector<DownloadPart> &parts, cudaStream_t st);

}  // namespace smax
