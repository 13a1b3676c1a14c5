// Drives staging.h's copies over the CPU runtime beside this file. argv[1]: the
// number of event creations that succeed before they start to fail.
#include "staging.h"

#include <cstdio>

static int check(cudaStream_t stream, size_t n, unsigned salt) {
    std::vector<char> host(n), device(n, 0), back(n, 0);
    for (size_t i = 0; i < n; i++) host[i] = (char)(i * 31 + i / 255 + salt + 1);
    if (rt::copy_to_device(0, stream, device.data(), host.data(), n) != cudaSuccess) return 1;
    if (device != host) return 2;   // the caller's next kernel would read this
    if (rt::copy_to_host(0, stream, back.data(), device.data(), n) != cudaSuccess) return 3;
    return back != host ? 4 : 0;
}

int main(int argc, char** argv) {
    if (argc > 1) fake::g.events_left = std::atoi(argv[1]);
    const size_t mib = size_t(1) << 20, sizes[] = {1, mib - 1, mib, mib + 1, 5 * mib + 7, 32 * mib, 33 * mib + 5};
    for (cudaStream_t stream : {cudaStream_t(7), cudaStreamPerThread})
        for (size_t n : sizes)
            if (int r = check(stream, n, 3)) return std::printf("stream %ld, %zu bytes: check %d\n", stream, n, r), 1;
    std::atomic<int> bad{0};
    std::vector<std::thread> callers;   // one finds the window in use and goes the plain way
    for (int k = 0; k < 4; k++)
        callers.emplace_back([&, k] {
            for (int i = 0; i < 4; i++) bad += check(k & 1 ? cudaStreamPerThread : 10 + k, 3 * mib + 11 * k, k);
        });
    for (std::thread& t : callers) t.join();
    if (bad) return std::printf("concurrent callers\n"), 1;
}
