#include "launch.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

namespace sg {

namespace {

struct Kernel {
    bool raised = false;
    std::map<std::pair<int, size_t>, int> ctas;   // per (threads, bytes): the driver's answer takes microseconds
};
std::mutex g_mu;
std::map<std::pair<int, const void *>, Kernel> g_kernels;   // per (device, kernel), guarded by g_mu

}  // namespace

int resident_ctas(const void *kern, int threads, size_t smem)
{
    // this thread's last answers: what they rest on, a raised limit and the
    // occupancy of a size, does not change (the lock and the maps cost a call of
    // seven launches 1 us)
    struct Answer {
        const void *kern;
        size_t smem;
        int dev, threads, n;
    };
    thread_local Answer answers[64];
    int dev = 0;
    cudaGetDevice(&dev);
    Answer &mine = answers[((uintptr_t)kern >> 4 ^ smem >> 4 ^ (size_t)dev) & 63];
    if (mine.kern == kern && mine.smem == smem && mine.threads == threads && mine.dev == dev) return mine.n;
    std::lock_guard<std::mutex> lk(g_mu);
    Kernel &k = g_kernels[{dev, kern}];
    if (!k.raised) {
        int most = 0;
        cudaFuncAttributes at{};
        k.raised = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
                   cudaFuncGetAttributes(&at, kern) == cudaSuccess &&
                   cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)at.sharedSizeBytes) ==
                       cudaSuccess;
    }
    auto it = k.ctas.find({threads, smem});
    int n = it != k.ctas.end() ? it->second : 0;
    if (n == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess) return 1;
        n = std::max(n, 1);
        if (k.ctas.size() >= 64) k.ctas.clear();
        k.ctas[{threads, smem}] = n;
    }
    if (k.raised) mine = {kern, smem, dev, threads, n};
    return n;
}

}  // namespace sg
