#include "launch.hpp"

#include <cuda_runtime.h>

#include <algorithm>
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
    int dev = 0;
    cudaGetDevice(&dev);
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
    if (it != k.ctas.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess) return 1;
    if (k.ctas.size() >= 64) k.ctas.clear();
    return k.ctas[{threads, smem}] = std::max(n, 1);
}

}  // namespace sg
