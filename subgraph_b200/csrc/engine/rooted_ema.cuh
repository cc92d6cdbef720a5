// The product step of the rooted rows: for every result set O (the relative
// colors of n - 1 vertices) the sum over its splits of main[M] * agg[O - M],
// in the order of the colors themselves.  A tile of vertices per CTA: the
// aggregate and main rows are read as they lie (coalesced) and land in shared
// memory transposed, each column at its rank in the colors' own order, where
// one index structure (|s|-1 vertices, mains of |main|-1, over k-1 colors)
// serves every vertex; results go back to the relative columns.
#pragma once
#include "launch.hpp"
#include "rooted.hpp"
#include "tile.cuh"

namespace sg {
namespace rt {

constexpr int kEmaThreads = 512;   // most threads a tile
// A tile that takes much of an SM's shared memory gets 512 threads, so that the
// few that fit still fill the SM's warps; a small one 256.
inline int ema_threads(size_t smem) { return smem > 36 * 1024 ? 512 : 256; }

// Rows to their places in shared memory, element by element (cp.async): all of
// a tile's elements are in flight together and hold no registers.
template <typename T>
__device__ __forceinline__ void ema_rows(const T *src, int pitch, const uint16_t *perm, int n, const uint8_t *color, int v0,
                                         int tv, T *dst, int RS)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t dst_s = (uint32_t)__cvta_generic_to_shared(dst);
    for (int vi = warp; vi < tv; vi += (int)blockDim.x / 32) {
        const T *row = src + (size_t)(v0 + vi) * pitch;
        const uint16_t *p = perm + (size_t)__ldg(color + v0 + vi) * n;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) {
            const uint32_t to = dst_s + (uint32_t)(((int)__ldg(p + j) * RS + vi) * (int)sizeof(T));
            if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(row + j) : "memory");
            else cp_async4_s(to, row + j);
        }
    }
}

template <typename T>
__device__ __forceinline__ void ema_store(const EmaArgs &a, const T *out_s, int RS, int v0, int tv)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int vi = warp; vi < tv; vi += (int)blockDim.x / 32) {
        T *row = reinterpret_cast<T *>(a.out) + (size_t)(v0 + vi) * a.out_pitch;
        const uint16_t *p = a.perm_o + (size_t)__ldg(a.color + v0 + vi) * a.nO;
#pragma unroll 4
        for (int j = lane; j < a.nO; j += 32) row[j] = out_s[(int)__ldg(p + j) * RS + vi];
    }
}

// the register-blocked schedule (blk_ema.cuh)
template <int N, int P> __global__ void __launch_bounds__(kEmaThreads) k_ema_blk(EmaArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int TV = a.tile_v, RS = TV + 1;
    float *agg_s = reinterpret_cast<float *>(smem_raw);
    float *main_s = agg_s + (size_t)a.nA * RS;
    float *out_s = main_s + (size_t)a.nM * RS;
    const int v0 = blockIdx.x * TV, tv = min(TV, a.V - v0);
    ema_rows(reinterpret_cast<const float *>(a.agg), a.agg_pitch, a.perm_a, a.nA, a.color, v0, tv, agg_s, RS);
    ema_rows(reinterpret_cast<const float *>(a.main), a.main_pitch, a.perm_m, a.nM, a.color, v0, tv, main_s, RS);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    StageDesc d{};
    d.blk = a.blk;
    d.blk_nblocks = a.blk_nblocks;
    blk::ema_blocks<N, P>(d, agg_s, main_s, out_s, RS, RS, TV, threadIdx.x >> 5, blockDim.x >> 5, threadIdx.x & 31);
    __syncthreads();
    ema_store(a, out_s, RS, v0, tv);
}

template <int N, int P> static void launch_ema_shape(const EmaArgs &a, size_t smem, cudaStream_t st)
{
    auto kern = k_ema_blk<N, P>;
    resident_ctas((const void *)kern, ema_threads(smem), smem);
    kern<<<(a.V + a.tile_v - 1) / a.tile_v, ema_threads(smem), smem, st>>>(a);
}

}  // namespace rt
}  // namespace sg
