// download.cu -- large device-to-host copies into fresh pageable memory.
//
// A copy into pageable memory that nobody has touched runs at the speed of one
// driver thread that also takes every page fault (2 GB/s here).  A large
// download is cut into pieces instead: a few host threads each copy their
// pieces into two pinned buffers, one arriving while the other is copied out,
// so the link stays busy and the faults, on 2 MB pages where the system
// allows, are taken by all of them.  A product of 13 M entries (160 MB) took
// 104 ms that way, including a second copy into numpy's memory, and
// takes 8.4 ms now; the link alone needs about 3 ms.  Below 4 MB a plain copy
// is as fast as starting the threads.
#include "download.cuh"

#include <sys/mman.h>

#include <algorithm>
#include <cstring>
#include <thread>

namespace smax {

bool DownloadStage::ensure() {
    if (ready || unfit) return ready;
    bool ok = cudaHostAlloc(&pinned, kPiece * 2 * kWorkers, cudaHostAllocDefault) == cudaSuccess;
    if (!ok) pinned = nullptr;
    ok = ok && cudaEventCreateWithFlags(&start, cudaEventDisableTiming) == cudaSuccess;
    for (int w = 0; w < kWorkers; ++w) {
        ok = ok && cudaStreamCreateWithFlags(&streams[w], cudaStreamNonBlocking) == cudaSuccess;
        for (int i = 0; i < 2; ++i)
            ok = ok && cudaEventCreateWithFlags(&done[w][i], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        (void)cudaGetLastError();
        release();
        unfit = true;  // downloads stay plain copies
    }
    return ready = ok;
}

void DownloadStage::release() {
    for (int w = 0; w < kWorkers; ++w) {
        if (streams[w]) cudaStreamDestroy(streams[w]);
        streams[w] = nullptr;
        for (int i = 0; i < 2; ++i) {
            if (done[w][i]) cudaEventDestroy(done[w][i]);
            done[w][i] = nullptr;
        }
    }
    if (start) cudaEventDestroy(start);
    start = nullptr;
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
    ready = false;
}

namespace {

// 2 MB pages for the part of [p, p + bytes) that can hold them; only a hint
void prefer_huge_pages(void *p, size_t bytes) {
    constexpr uintptr_t kHuge = 2u << 20;
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + kHuge - 1) & ~(kHuge - 1);
    const uintptr_t b = (reinterpret_cast<uintptr_t>(p) + bytes) & ~(kHuge - 1);
    if (b > a) madvise(reinterpret_cast<void *>(a), b - a, MADV_HUGEPAGE);
}

}  // namespace

void download(DownloadStage &stage, const std::vector<DownloadPart> &parts, cudaStream_t st) {
    size_t total = 0;
    for (const DownloadPart &p : parts) total += p.bytes;
    if (total < DownloadStage::kLarge || !stage.ensure()) {
        for (const DownloadPart &p : parts)
            if (p.bytes) SMAX_CUDA(cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, st));
        SMAX_CUDA(cudaStreamSynchronize(st));
        return;
    }
    std::vector<DownloadPart> pieces;
    for (const DownloadPart &p : parts) {
        prefer_huge_pages(p.dst, p.bytes);
        for (size_t o = 0; o < p.bytes; o += DownloadStage::kPiece)
            pieces.push_back({static_cast<char *>(p.dst) + o, static_cast<const char *>(p.src) + o,
                              std::min(DownloadStage::kPiece, p.bytes - o)});
    }
    int device = 0;
    SMAX_CUDA(cudaGetDevice(&device));
    SMAX_CUDA(cudaEventRecord(stage.start, st));
    constexpr int W = DownloadStage::kWorkers;
    cudaError_t failed[W];
    auto work = [&](int w) {
        auto run = [&]() -> cudaError_t {
            cudaError_t e = cudaSetDevice(device);
            if (e != cudaSuccess) return e;
            cudaStream_t s = stage.streams[w];
            if ((e = cudaStreamWaitEvent(s, stage.start, 0)) != cudaSuccess) return e;
            char *buf[2] = {static_cast<char *>(stage.pinned) + DownloadStage::kPiece * (2 * w),
                            static_cast<char *>(stage.pinned) + DownloadStage::kPiece * (2 * w + 1)};
            auto fetch = [&](size_t i, int b) {
                cudaError_t r = cudaMemcpyAsync(buf[b], pieces[i].src, pieces[i].bytes, cudaMemcpyDeviceToHost, s);
                return r == cudaSuccess ? cudaEventRecord(stage.done[w][b], s) : r;
            };
            int b = 0;
            if ((size_t)w < pieces.size() && (e = fetch(w, 0)) != cudaSuccess) return e;
            for (size_t i = w; i < pieces.size(); i += W, b ^= 1) {
                if (i + W < pieces.size() && (e = fetch(i + W, b ^ 1)) != cudaSuccess) return e;
                if ((e = cudaEventSynchronize(stage.done[w][b])) != cudaSuccess) return e;
                std::memcpy(pieces[i].dst, buf[b], pieces[i].bytes);
            }
            return cudaSuccess;
        };
        failed[w] = run();
        // nothing of this thread stays in flight into the staging buffers
        if (failed[w] != cudaSuccess) cudaStreamSynchronize(stage.streams[w]);
    };
    // pieces of a thread that could not be started are copied by this one
    std::vector<std::thread> threads;
    int started = 1;
    try {
        for (; started < W; ++started) threads.emplace_back(work, started);
    } catch (...) {
    }
    work(0);
    for (int w = started; w < W; ++w) work(w);
    for (std::thread &t : threads) t.join();
    for (int w = 0; w < W; ++w) cuda_check(failed[w], "download");
}

}  // namespace smax
