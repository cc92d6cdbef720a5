// The product step of the rooted rows: the split loop (shapes without a block
// schedule, FP64 tables), the root step, and the dispatch (rooted_ema.cuh).
#include "rooted_ema.cuh"

namespace sg {
namespace rt {

__device__ __forceinline__ float product(float acc, float x, float y, bool fused)
{
    return fused ? __fmaf_rn(x, y, acc) : __fadd_rn(acc, __fmul_rn(x, y));
}
__device__ __forceinline__ double product(double acc, double x, double y, bool) { return __dadd_rn(acc, __dmul_rn(x, y)); }

template <typename T, bool FUSED> __global__ void __launch_bounds__(kEmaThreads) k_ema(EmaArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int TV = a.tile_v, RS = TV + 1;
    T *agg_s = reinterpret_cast<T *>(smem_raw);
    T *main_s = agg_s + (size_t)a.nA * RS;
    T *out_s = main_s + (size_t)a.nM * RS;
    const int v0 = blockIdx.x * TV, tv = min(TV, a.V - v0);
    ema_rows(reinterpret_cast<const T *>(a.agg), a.agg_pitch, a.perm_a, a.nA, a.color, v0, tv, agg_s, RS);
    ema_rows(reinterpret_cast<const T *>(a.main), a.main_pitch, a.perm_m, a.nM, a.color, v0, tv, main_s, RS);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (a.is_root) {
        if (warp != 0) return;
        // one warp: lane = vertex, its products summed in FP64 in split order
        double racc = 0.0;
        if (lane < tv) {
            for (int j = 0; j < a.S; ++j) {
                const uint32_t pk = __ldg(a.split + (size_t)j * a.split_stride);
                const T x = main_s[(pk & 0xffffu) * RS + lane], y = agg_s[(pk >> 16) * RS + lane];
                if (sizeof(T) == 8) racc = __dadd_rn(racc, __dmul_rn((double)y, (double)x));
                else racc = __dadd_rn(racc, (double)__fmul_rn((float)y, (float)x));
            }
            a.root_value[v0 + lane] = racc;
        }
        return;
    }
    // lanes = vertices (32 / TV outputs groups a warp), four result columns a
    // lane: four independent chains in split order
    const int vi = lane % TV, sub = lane / TV, per = 32 / TV;
    const int ng = (a.nO + 3) / 4;
    for (int g = warp * per + sub; g < ng; g += (int)(blockDim.x >> 5) * per) {
        const uint4 *sp = reinterpret_cast<const uint4 *>(a.split) + g;
        const int step = a.split_stride / 4;
        T c0 = T(0), c1 = T(0), c2 = T(0), c3 = T(0);
#pragma unroll 4
        for (int j = 0; j < a.S; ++j) {
            const uint4 pk = __ldg(sp + (size_t)j * step);
            c0 = product(c0, agg_s[(pk.x >> 16) * RS + vi], main_s[(pk.x & 0xffffu) * RS + vi], FUSED);
            c1 = product(c1, agg_s[(pk.y >> 16) * RS + vi], main_s[(pk.y & 0xffffu) * RS + vi], FUSED);
            c2 = product(c2, agg_s[(pk.z >> 16) * RS + vi], main_s[(pk.z & 0xffffu) * RS + vi], FUSED);
            c3 = product(c3, agg_s[(pk.w >> 16) * RS + vi], main_s[(pk.w & 0xffffu) * RS + vi], FUSED);
        }
        const T c[4] = {c0, c1, c2, c3};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (4 * g + i < a.nO) out_s[(4 * g + i) * RS + vi] = c[i];
    }
    __syncthreads();
    ema_store(a, out_s, RS, v0, tv);
}

static size_t ema_smem(int nA, int nM, int nO, int tv, size_t es, bool root)
{
    return ((size_t)(nA + nM + (root ? 0 : nO)) * (tv + 1)) * es;
}

int ema_tile(int nA, int nM, int nO, bool fp64, bool root, bool blocked)
{
    const size_t es = fp64 ? 8 : 4;
    const int least = blocked ? 16 : 8;
    for (size_t limit : {72 * 1024, 113 * 1024, 225 * 1024})
        for (int tv = 32; tv >= least; tv /= 2)
            if (ema_smem(nA, nM, nO, tv, es, root) <= limit) return tv;
    return 0;
}

bool launch_ema_a(const EmaArgs &a, size_t smem, cudaStream_t st);
bool launch_ema_b(const EmaArgs &a, size_t smem, cudaStream_t st);
bool launch_ema_c(const EmaArgs &a, size_t smem, cudaStream_t st);
bool launch_ema_d(const EmaArgs &a, size_t smem, cudaStream_t st);
bool launch_ema_e(const EmaArgs &a, size_t smem, cudaStream_t st);

void launch_ema(const EmaArgs &a0, bool fp64, cudaStream_t st)
{
    EmaArgs a = a0;
    if (a.V <= 0) return;
    if (!fp64 && a.blk && !a.is_root) {
        a.tile_v = ema_tile(a.nA, a.nM, a.nO, false, false, true);
        if (a.tile_v > 0) {
            const size_t smem = ema_smem(a.nA, a.nM, a.nO, a.tile_v, 4, false);
            if (launch_ema_a(a, smem, st) || launch_ema_b(a, smem, st) || launch_ema_c(a, smem, st) ||
                launch_ema_d(a, smem, st) || launch_ema_e(a, smem, st))
                return;
        }
    }
    a.tile_v = ema_tile(a.nA, a.nM, a.nO, fp64, a.is_root, false);
    const size_t smem = ema_smem(a.nA, a.nM, a.nO, a.tile_v, fp64 ? 8 : 4, a.is_root);
    const int tiles = (a.V + a.tile_v - 1) / a.tile_v;
    auto go = [&](auto kern) {
        const int threads = a.is_root ? 128 : ema_threads(smem);
        resident_ctas((const void *)kern, threads, smem);
        kern<<<tiles, threads, smem, st>>>(a);
    };
    if (fp64) go(k_ema<double, false>);
    else if (a.fused) go(k_ema<float, true>);
    else go(k_ema<float, false>);
}

}  // namespace rt
}  // namespace sg
