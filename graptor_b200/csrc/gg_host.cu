// gg_host.cu -- results to the caller's host memory.
//
// A copy into pageable memory (a fresh numpy array, a std::vector) goes
// through the driver's staging buffer on one thread, which also takes the
// destination's page faults: 5 to 7 GB/s measured, where the link gives 55.
// Here several threads of the call copy pieces in turn: each has two
// page-locked slots, one filling from the device while it empties the other
// into the destination (and faults its pages in).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

#include "gg_internal.cuh"

namespace gg {

constexpr size_t kPiece = 1u << 20;     // bytes per slot
constexpr int kMaxCopiers = 8;          // threads; 16 MiB page-locked per context
// From here on threads: below, starting them costs what they save (mean of 100
// copies into memory that has its pages, directly -> by threads: 4 MiB 275 -> 340
// us, 6 MiB 387 -> 415, 8 MiB 500 -> 505, 12 MiB 745 -> 690, 16 MiB 975 -> 815, 24 MiB
// 1450 -> 960; into fresh pages 64 MiB 13400 -> 3400).
constexpr size_t kStagedBytes = 8u << 20;

void host_stage_free(gg_ctx *ctx) {
    for (auto &e : ctx->stage_ev) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    cudaFreeHost(ctx->stage);
    ctx->stage = nullptr;
}

// The context's device as the calling thread's current one, whose own comes
// back at the end: the slots' events belong to it, and a download leaves the
// caller's device as it is.
struct CurrentDevice {
    int before = -1;
    explicit CurrentDevice(int device) {
        if (cudaGetDevice(&before) != cudaSuccess || before == device) before = -1;
        else cudaSetDevice(device);
    }
    ~CurrentDevice() {
        if (before >= 0) cudaSetDevice(before);
    }
};

static bool host_stage(gg_ctx *ctx) {
    if (ctx->stage) return true;
    bool ok = cudaHostAlloc(&ctx->stage, 2 * kMaxCopiers * kPiece, cudaHostAllocDefault) == cudaSuccess;
    for (auto &e : ctx->stage_ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        host_stage_free(ctx);
    }
    return ok;
}

static gg_status direct(gg_ctx *ctx, void *dst, const void *src, size_t bytes) {
    GG_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    GG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return GG_OK;
}

// bytes of device memory to host memory, after the work on the context's
// stream; returns when they are there.
gg_status host_download(gg_ctx *ctx, void *dst, const void *src, size_t bytes) {
    const CurrentDevice device(ctx->device);
    if (bytes == 0) return direct(ctx, dst, src, 0);
    cudaPointerAttributes at;
    const bool known = cudaPointerGetAttributes(&at, dst) == cudaSuccess;
    cudaGetLastError();
    const bool pageable = known && at.type == cudaMemoryTypeUnregistered;
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const int T = (int)std::min<size_t>(std::min<size_t>(kMaxCopiers, cores), bytes / (2 * kPiece));
    if (!pageable || bytes < kStagedBytes || T < 2 || !host_stage(ctx)) return direct(ctx, dst, src, bytes);
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    std::atomic<int> failed{(int)cudaSuccess};
    // copier w takes pieces w, w + T, ...
    auto copier = [&](int w) {
        cudaError_t e = cudaSetDevice(ctx->device);
        auto slot = [&](size_t k) { return (char *)ctx->stage + (2 * w + (k & 1)) * kPiece; };
        auto fill = [&](size_t k) {  // this copier's k-th piece
            const size_t at = (w + k * T) * kPiece;
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(slot(k), (const char *)src + at, std::min(kPiece, bytes - at),
                                    cudaMemcpyDeviceToHost, ctx->stream);
            if (e == cudaSuccess) e = cudaEventRecord(ctx->stage_ev[2 * w + (k & 1)], ctx->stream);
        };
        const size_t mine = (size_t)w < pieces ? (pieces - w + T - 1) / T : 0;
        if (mine) fill(0);
        for (size_t k = 0; k < mine && e == cudaSuccess; ++k) {
            if (k + 1 < mine) fill(k + 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(ctx->stage_ev[2 * w + (k & 1)]);
            const size_t to = (w + k * T) * kPiece;
            if (e == cudaSuccess) std::memcpy((char *)dst + to, slot(k), std::min(kPiece, bytes - to));
        }
        if (e != cudaSuccess) failed = (int)e;
    };
    std::vector<std::thread> threads;
    int started = 1;  // copier 0 is this thread
    try {
        threads.reserve(T);
        for (; started < T; ++started) threads.emplace_back(copier, started);
    } catch (const std::exception &) {  // no more threads: their shares are taken here
    }
    copier(0);
    for (int w = started; w < T; ++w) copier(w);
    for (auto &t : threads) t.join();
    const cudaError_t e = (cudaError_t)failed.load();
    if (e != cudaSuccess) {
        cudaStreamSynchronize(ctx->stream);  // nothing still writes the slots
        return cuda_error(ctx, e, "download");
    }
    return GG_OK;
}

}  // namespace gg
