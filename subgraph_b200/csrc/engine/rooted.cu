// Kernels of the rooted-row steps (rooted.hpp): neighbour colors and counts,
// the gather of neighbour rows, the root step of a one-hot main.
#include "rooted.hpp"

#include <algorithm>

#include "tile.cuh"

namespace sg {
namespace rt {

namespace {

constexpr int kEdgeThreads = 256;

}  // namespace

// ---------------------------------------------------------------------------
// Per coloring: every neighbour entry's color relative to its vertex, and the
// vertex's neighbour count of each relative color (the rows of a
// sub-template of two vertices, exact integers in any order).  A block's
// threads take one hub, or 8 vertices at a warp each, 32 at 8 threads each, or
// 128 of at most eight neighbours at 2 threads each (8 threads of which most had
// nothing to do took 62 us at 10^6 vertices of degree 4).
// ---------------------------------------------------------------------------
template <typename T, int G>
__device__ __forceinline__ void edge_rows(const EdgeArgs &a, int v, int t, unsigned *cnt)
{
    const int b = a.color[v];
    const int beg = __ldg(a.off + v), end = __ldg(a.off + v + 1);
    for (int e0 = beg; e0 < end; e0 += 4 * G) {
        int u[4], c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) u[i] = e0 + i * G + t < end ? __ldg(a.adj + e0 + i * G + t) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = u[i] >= 0 ? (int)__ldg(a.color + u[i]) : 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (u[i] < 0) continue;
            const int d = c[i] - b + (c[i] < b ? a.k : 0);
            atomicAdd(cnt + d, 1u);
            if (a.adjd) a.adjd[e0 + i * G + t] = u[i] < a.lim ? (int32_t)((uint32_t)u[i] | (uint32_t)d << 28) : 0;
        }
    }
}

// A vertex's row by its G threads, an element each; by two threads in pieces of 16
// bytes, of which rows are whole ones.  (Pieces by eight threads leave most of
// them idle: the kernel 14.2 us against 13.4, P3 on R-MAT scale 16.)
template <typename T, int G> __device__ __forceinline__ void count_row(const EdgeArgs &a, int v, int t, const unsigned *cnt)
{
    constexpr int E = G == 2 ? 16 / (int)sizeof(T) : 1;
    for (int j = t * E; j < a.cnt_pitch; j += G * E) {
        __align__(16) T x[E], y[E];
#pragma unroll
        for (int i = 0; i < E; ++i) {
            x[i] = j + i < a.k - 1 ? (T)cnt[j + i + 1] : T(0);
            y[i] = leaf_value(x[i], true);
        }
        T *o = reinterpret_cast<T *>(a.cnt) + (size_t)v * a.cnt_pitch + j;
        T *so = reinterpret_cast<T *>(a.scnt) + (size_t)v * a.cnt_pitch + j;
        if constexpr (E == 1) {
            *o = x[0];
            if (a.scnt) *so = y[0];
        } else {
            *reinterpret_cast<uint4 *>(o) = *reinterpret_cast<uint4 *>(x);
            if (a.scnt) *reinterpret_cast<uint4 *>(so) = *reinterpret_cast<uint4 *>(y);
        }
    }
}

// G threads a vertex, the block's vertices from v0
template <typename T, int G>
__device__ __forceinline__ void edge_group(const EdgeArgs &a, int v0, int end, unsigned *cnt_s)
{
    const int g = threadIdx.x / G, t = threadIdx.x % G, v = v0 + g;
    if (v < end) edge_rows<T, G>(a, v, t, cnt_s + g * 17);
    __syncwarp();
    if (v < end) count_row<T, G>(a, v, t, cnt_s + g * 17);
}

template <typename T> __global__ void __launch_bounds__(kEdgeThreads) k_edges(EdgeArgs a, int mid, int low, int nb_mid, int nb_8)
{
    extern __shared__ unsigned cnt_s[];   // [most vertices of a block][17]
    int blk = blockIdx.x;
    const int rows = blk < a.hubs + nb_mid ? kEdgeThreads / 32 : blk < a.hubs + nb_mid + nb_8 ? kEdgeThreads / 8 : kEdgeThreads / 2;
    for (int i = threadIdx.x; i < rows * 17; i += kEdgeThreads) cnt_s[i] = 0;
    __syncthreads();
    if (blk < a.hubs) {
        // counters of a warp each, then their sum
        unsigned *mine = cnt_s + (threadIdx.x >> 5) * 17;
        edge_rows<T, kEdgeThreads>(a, blk, threadIdx.x, mine);
        __syncthreads();
        if (threadIdx.x < 17) {
            unsigned s = 0;
            for (int w = 0; w < kEdgeThreads / 32; ++w) s += cnt_s[w * 17 + threadIdx.x];
            cnt_s[threadIdx.x] = s;
        }
        __syncthreads();
        count_row<T, kEdgeThreads>(a, blk, threadIdx.x, cnt_s);
        return;
    }
    blk -= a.hubs;
    if (blk < nb_mid) return edge_group<T, 32>(a, a.hubs + blk * (kEdgeThreads / 32), mid, cnt_s);
    blk -= nb_mid;
    if (blk < nb_8) return edge_group<T, 8>(a, mid + blk * (kEdgeThreads / 8), low, cnt_s);
    edge_group<T, 2>(a, low + (blk - nb_8) * (kEdgeThreads / 2), a.V1, cnt_s);
}

void launch_edges(const EdgeArgs &a, int32_t mid, int32_t low, bool fp64, cudaStream_t st)
{
    if (a.V1 <= 0) return;
    const int nb_mid = (mid - a.hubs + kEdgeThreads / 32 - 1) / (kEdgeThreads / 32);
    const int nb_8 = (low - mid + kEdgeThreads / 8 - 1) / (kEdgeThreads / 8);
    const int nb_2 = (a.V1 - low + kEdgeThreads / 2 - 1) / (kEdgeThreads / 2);
    const int grid = a.hubs + nb_mid + nb_8 + nb_2;
    // a block's counters (below the 48 KB any kernel may have); what an SM's blocks
    // do not take is cache for the colors
    const size_t smem = (size_t)kEdgeThreads / (nb_2 > 0 ? 2 : 8) * 17 * sizeof(unsigned);
    if (fp64) k_edges<double><<<grid, kEdgeThreads, smem, st>>>(a, mid, low, nb_mid, nb_8);
    else k_edges<float><<<grid, kEdgeThreads, smem, st>>>(a, mid, low, nb_mid, nb_8);
}

bool gather_fits(int k, int nA, int nR, bool fp64)
{
    // row offsets in 16 bits (13 beside a slot's member), a counter per column block
    // (of 128 slots at least; more than 128 columns, the narrower ones take one)
    return k <= 16 && nR < 0x1fff && (size_t)nR * (fp64 ? 8 : 4) + 32 < 0xffff && nA <= 128 * kColumnBlocks;
}

int gather_lanes(const GatherArgs &a) { return a.slots <= 1 ? 1 : a.slots <= 4 ? 4 : a.slots <= 8 ? 8 : a.slots <= 16 ? 16 : 32; }

int launch_gather(const GatherArgs &a, bool fp64, int sm_count, cudaStream_t st)
{
    if (a.map.n == 0 && a.hubs == 0) return 0;
    if (fp64) launch_gather_f64(a, sm_count, st);
    else launch_gather_f32(a, sm_count, st);
    return 1;
}

// ---------------------------------------------------------------------------
// The root's values summed over tiles of tile_v vertices, one warp a tile, in
// the general path's order (fused_tile: a lane's vertices one after another,
// then the lanes by halves); with a one-hot main the aggregate is the value.
// ---------------------------------------------------------------------------
template <typename T> __global__ void __launch_bounds__(256) k_root_tiles(RootArgs a)
{
    const T *val = reinterpret_cast<const T *>(a.val);
    const int lane = threadIdx.x & 31, tile = (int)(blockIdx.x * 8 + (threadIdx.x >> 5));
    if ((int64_t)tile * a.tile_v >= a.V1) return;
    const int v0 = tile * a.tile_v, v1 = min(v0 + a.tile_v, a.V1);
    double s = 0.0;
    for (int v = v0 + lane; v < v1; v += 32) {
        const double x = (double)val[(size_t)v * a.pitch];
        if (a.root_vertex) a.root_vertex[v] = x;
        s = __dadd_rn(s, x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(0xffffffffu, s, o));
    if (lane == 0) a.root_partial[tile] = s;
}

int launch_root_tiles(const RootArgs &a, bool fp64, cudaStream_t st)
{
    const int tiles = (a.V1 + a.tile_v - 1) / a.tile_v;
    if (tiles == 0) return 0;
    if (fp64) k_root_tiles<double><<<(tiles + 7) / 8, 256, 0, st>>>(a);
    else k_root_tiles<float><<<(tiles + 7) / 8, 256, 0, st>>>(a);
    return tiles;
}

}  // namespace rt
}  // namespace sg
