#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace rt {

// ---------------------------------------------------------------------------
// Large copies between the device and a caller's pageable memory. The driver
// stages such a copy through its own pinned buffers on one host thread, which
// also takes the page faults of a fresh destination: a full-HD film (25 MB) took
// 4 to 8 ms each way, the link needs 0.5. Here four threads move the chunks of
// a pinned window (one per device, 32 MiB, kept) while the next ones are on the
// link. A copy below 1 MiB, or one that finds the window in use by another
// thread's call, goes the driver's way. Both return with the copy done.
// Every thread waits for the copies that it queued: with cudaStreamPerThread
// each names a stream of its own, which the caller's wait does not cover.
// ---------------------------------------------------------------------------
constexpr size_t kStageChunk = size_t(1) << 20, kStageChunks = 32;
constexpr int kStageThreads = 4;
struct Stage {
    std::mutex mu;
    char* mem = nullptr;
    cudaEvent_t landed[kStageChunks] = {};
    // With mu held, which a copy holds until it is done.
    void release() {
        for (cudaEvent_t& e : landed) {
            if (e) cudaEventDestroy(e);
            e = {};
        }
        if (mem) cudaFreeHost(mem);
        mem = nullptr;
    }
};
inline Stage g_stage[16];

inline cudaError_t stage_copy(int dev, cudaStream_t stream, char* host, char* device, size_t n, bool to_host) {
    auto plain = [&] {
        cudaError_t e = to_host ? cudaMemcpyAsync(host, device, n, cudaMemcpyDeviceToHost, stream)
                                : cudaMemcpyAsync(device, host, n, cudaMemcpyHostToDevice, stream);
        return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
    };
    if (n < kStageChunk || dev < 0 || dev >= 16) return plain();
    cudaPointerAttributes at_host{};
    if (cudaPointerGetAttributes(&at_host, host) == cudaSuccess && at_host.type != cudaMemoryTypeUnregistered)
        return plain();   // pinned or device-accessible memory: the link takes it as it is
    Stage& st = g_stage[dev];
    std::unique_lock<std::mutex> lk(st.mu, std::try_to_lock);
    if (!lk.owns_lock()) return plain();
    if (!st.mem) {   // no window or no events: the driver's way
        bool ok = cudaMallocHost(&st.mem, kStageChunk * kStageChunks) == cudaSuccess;
        if (!ok) st.mem = nullptr;
        for (size_t c = 0; ok && c < kStageChunks; c++) {
            ok = cudaEventCreateWithFlags(&st.landed[c], cudaEventDisableTiming) == cudaSuccess;
            if (!ok) st.landed[c] = {};
        }
        if (!ok) {
            cudaGetLastError();
            st.release();
            return plain();
        }
    }
    for (size_t w = 0; w < n; w += kStageChunk * kStageChunks) {   // one window at a time
        const size_t bytes = std::min(n - w, kStageChunk * kStageChunks);
        const size_t chunks = (bytes + kStageChunk - 1) / kStageChunk;
        std::atomic<int> err{cudaSuccess};
        auto note = [&](cudaError_t e) {
            int none = cudaSuccess;
            if (e != cudaSuccess) err.compare_exchange_strong(none, e);
        };
        auto len = [&](size_t c) { return std::min(kStageChunk, bytes - c * kStageChunk); };
        if (to_host)
            for (size_t c = 0; c < chunks; c++) {
                note(cudaMemcpyAsync(st.mem + c * kStageChunk, device + w + c * kStageChunk, len(c),
                                     cudaMemcpyDeviceToHost, stream));
                note(cudaEventRecord(st.landed[c], stream));
            }
        std::atomic<size_t> at{0};
        auto work = [&] {
            cudaSetDevice(dev);
            for (size_t c; (c = at.fetch_add(1)) < chunks;) {
                char *mine = st.mem + c * kStageChunk, *theirs = host + w + c * kStageChunk;
                if (to_host) {
                    note(cudaEventSynchronize(st.landed[c]));
                    std::memcpy(theirs, mine, len(c));
                } else {
                    std::memcpy(mine, theirs, len(c));
                    note(cudaMemcpyAsync(device + w + c * kStageChunk, mine, len(c), cudaMemcpyHostToDevice, stream));
                }
            }
            if (!to_host) note(cudaStreamSynchronize(stream));
        };
        std::vector<std::thread> pool;
        try {
            for (size_t k = 1; k < std::min<size_t>(kStageThreads, chunks); k++) pool.emplace_back(work);
        } catch (const std::exception&) {   // no more threads: this one does the rest
        }
        work();
        for (std::thread& t : pool) t.join();
        note(cudaStreamSynchronize(stream));   // before the window is used again
        if (err != cudaSuccess) return static_cast<cudaError_t>(err.load());
    }
    return cudaSuccess;
}
inline cudaError_t copy_to_host(int dev, cudaStream_t stream, void* dst, const void* src, size_t n) {
    return stage_copy(dev, stream, static_cast<char*>(dst), static_cast<char*>(const_cast<void*>(src)), n, true);
}
inline cudaError_t copy_to_device(int dev, cudaStream_t stream, void* dst, const void* src, size_t n) {
    return stage_copy(dev, stream, static_cast<char*>(const_cast<void*>(src)), static_cast<char*>(dst), n, false);
}

}  // namespace rt
