// The few CUDA runtime calls that staging.h makes, on the CPU, with the
// asynchrony that matters to it: a copy from or to pinned memory is done when its
// stream is waited for (or an event behind it) and not before, and
// cudaStreamPerThread is another stream in each thread. A stream that nobody
// waits for never runs.
#pragma once

#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <set>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaEventDisableTiming = 2 };
struct cudaPointerAttributes {
    cudaMemoryType type;
};
using cudaStream_t = long;
using cudaEvent_t = long;
constexpr cudaStream_t cudaStreamPerThread = 2;

namespace fake {
struct State {
    std::recursive_mutex mu;
    std::map<long, std::deque<std::function<void()>>> queues;
    std::map<long, std::pair<long, size_t>> events;   // the stream and how much of it lies before the event
    std::map<long, size_t> done;                      // per stream: operations run
    std::set<char*> pinned;
    long next_event = 1, next_thread = 100;
    int events_left = 1 << 30;   // event creations that still succeed
};
inline State g;
inline long key(cudaStream_t s) {
    thread_local long mine = 0;
    if (s != cudaStreamPerThread) return s;
    if (!mine) mine = g.next_thread++;
    return mine;
}
inline bool is_pinned(const void* p) {
    auto it = g.pinned.upper_bound((char*)p);
    return it != g.pinned.begin() && (const char*)p < *--it + (size_t(32) << 20);
}
inline void run(long k, size_t upto) {
    auto& q = g.queues[k];
    while (!q.empty() && g.done[k] < upto) {
        q.front()();
        q.pop_front();
        g.done[k]++;
    }
}
}  // namespace fake

inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    a->type = fake::is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
template <class T>
cudaError_t cudaMallocHost(T** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    *p = (T*)std::malloc(n);
    fake::g.pinned.insert((char*)*p);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    fake::g.pinned.erase((char*)p);
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    fake::run(fake::key(s), size_t(-1));
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    long k = fake::key(s);
    bool later = fake::is_pinned(dst) || fake::is_pinned(src);
    fake::g.queues[k].push_back([=] { std::memcpy(dst, src, n); });
    if (!later) fake::run(k, size_t(-1));   // pageable memory: through the driver's own buffers
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    if (fake::g.events_left-- <= 0) return cudaErrorMemoryAllocation;
    *e = fake::g.next_event++;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    if (!e) return cudaErrorInvalidValue;
    long k = fake::key(s);
    fake::g.events[e] = {k, fake::g.done[k] + fake::g.queues[k].size()};
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(fake::g.mu);
    if (!e) return cudaErrorInvalidValue;
    auto [k, upto] = fake::g.events[e];
    fake::run(k, upto);
    return cudaSuccess;
}
