// Device side of the rooted rows' gather (rooted.hpp), instantiated for FP32
// and FP64 tables in rooted_gather_f32.cu and rooted_gather_f64.cu.
#pragma once
#include <algorithm>

#include "launch.hpp"
#include "rooted.hpp"
#include "tile.cuh"

namespace sg {
namespace rt {

namespace {

// The chunk of ticket t: its first vertex and one past its last.
__device__ __forceinline__ bool chunk_of(const ChunkMap &m, int t, int &v0, int &v1)
{
    int c = 0;
    while (c < m.n && t >= m.base[c + 1]) ++c;
    if (c >= m.n) return false;
    v0 = m.first[c] + (t - m.base[c]) * m.per[c];
    v1 = min(v0 + m.per[c], m.first[c + 1]);
    return true;
}

}  // namespace

// ---------------------------------------------------------------------------
// The gather: every vertex's sums of its neighbours' rows, at the color sets
// without its own color, in list order.  Three parts:
//   hubs    a CTA per (vertex, columns), the longest lists first;
//   wide    a warp per run of vertices, R sums a lane, rows staged in shared
//           memory by 16-byte asynchronous copies (cp.async);
//   narrow  G lanes a vertex, R sums a lane, rows read where they lie.
// One kernel takes the hubs first and then the wide or the narrow part, so
// that the longest chains run beside the other vertices.
// ---------------------------------------------------------------------------
constexpr int kWarps = 8, kGatherThreads = 32 * kWarps;

template <typename T> __device__ __forceinline__ void cp_async_elem(uint32_t dst, const void *src, uint32_t n)
{
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else
        cp_async4_zs(dst, src, n);
}

// Hubs.  A column's sum over its list is one chain of dependent adds, four
// cycles each, so one warp does nothing but add: lane l reads column l of
// batch after batch of neighbours from shared memory.  The other warps fill
// the batches two ahead, 32 / GH neighbours at a time: a lane copies
// (cp.async) the one element of the neighbour's row that its column takes, or
// zeros.
constexpr int kHubStages = 3;
template <int GH> constexpr int hub_fills() { return GH == 1 ? 4 : 16; }   // a producer warp and batch
template <typename T, int GH> constexpr size_t hub_bytes() { return (size_t)kHubStages * (kWarps - 1) * hub_fills<GH>() * 32 * sizeof(T); }

// Whether a CTA takes hub items (asked by its thread 0).  The CTAs of an SM start
// together and would take the first items, the longest lists, side by side:
// 20 lists of 100,000 neighbours ran on five SMs, four on each, at 19 cycles a
// neighbour.  Where that is the kernel's time (launch_gather's caller says so)
// only the first CTA of an SM takes items, until none is left.
__device__ __forceinline__ bool hub_turn(const GatherArgs &a)
{
    if (a.hubs == 0) return false;
    if (!a.spread) return true;
    uint32_t sm;
    asm("mov.u32 %0, %%smid;" : "=r"(sm));
    sm %= 32 * kSmWords;
    const uint32_t bit = 1u << (sm & 31);
    return !(atomicOr(a.sm_seen + (sm >> 5), bit) & bit);
}

template <typename T, int GH> __device__ __forceinline__ void hub_part(const GatherArgs &a, unsigned char *smem)
{
    constexpr int NPF = 32 / GH, PER = hub_fills<GH>(); // neighbours a fill, fills
    constexpr int NPW = PER * NPF;                  // neighbours a producer and batch
    constexpr int NB = (kWarps - 1) * NPW;              // neighbours a batch
    constexpr int NWD = (NPW + 31) / 32;                // words a lane holds of them
    T *xs = reinterpret_cast<T *>(smem);                // [kHubStages][NB][GH]
    __shared__ uint16_t tab[16 * GH];
    __shared__ int s_item;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lg = lane % GH, sub = lane / GH;
    const int nblk = (a.nA + GH - 1) / GH;
    const char *aux = reinterpret_cast<const char *>(a.aux);
    const uint32_t row_bytes = (uint32_t)a.pitch * (uint32_t)sizeof(T);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(a.hub_ticket, 1);
        __syncthreads();
        const int v = s_item / nblk, col0 = (s_item - v * nblk) * GH;
        if (v >= a.hubs) break;
        for (int i = threadIdx.x; i < a.k * GH; i += kGatherThreads) {
            const int d = i / GH, j = col0 + i % GH;
            tab[i] = d > 0 && j < a.nA ? __ldg(a.idx + (size_t)(d - 1) * a.nA + j) : (uint16_t)0xffffu;
        }
        const int beg = __ldg(a.off + v), deg = __ldg(a.off + v + 1) - beg;
        const int nbt = (deg + NB - 1) / NB;
        __syncthreads();
        if (warp < kWarps - 1) {
            const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(xs) + (uint32_t)((warp * NPW * GH + lane) * sizeof(T));
            auto words = [&](int b, uint32_t(&w)[NWD]) {
#pragma unroll
                for (int i = 0; i < NWD; ++i) {
                    const int e = b * NB + warp * NPW + i * 32 + (NPW < 32 ? lane & (NPW - 1) : lane);
                    w[i] = e < deg ? (uint32_t)__ldg(a.adjd + beg + e) : 0u;
                }
            };
            auto fill = [&](int b, const uint32_t(&w)[NWD]) {
                const uint32_t dst = dst0 + (uint32_t)((b % kHubStages) * (NB * GH * (int)sizeof(T)));
                // the shuffles and table reads of eight fills, then their copies
#pragma unroll
                for (int i0 = 0; i0 < PER; i0 += 8) {
                    constexpr int Q = PER < 8 ? PER : 8;
                    uint32_t x[Q], c[Q];
#pragma unroll
                    for (int i = 0; i < Q; ++i)
                        x[i] = GH == 1 ? w[(i0 + i) * NPF / 32] : __shfl_sync(0xffffffffu, w[(i0 + i) * NPF / 32], ((i0 + i) * NPF) % 32 + sub);
#pragma unroll
                    for (int i = 0; i < Q; ++i) c[i] = tab[(x[i] >> 28) * GH + lg];
#pragma unroll
                    for (int i = 0; i < Q; ++i) {
                        const bool hit = c[i] != 0xffffu;
                        const char *src = aux + (uint64_t)(x[i] & 0x0fffffffu) * row_bytes + (hit ? c[i] : 0u) * (uint32_t)sizeof(T);
                        cp_async_elem<T>(dst + (uint32_t)((i0 + i) * 32 * sizeof(T)), src, hit ? (uint32_t)sizeof(T) : 0u);
                    }
                }
            };
            uint32_t w0[NWD], w1[NWD], w2[NWD];
            words(0, w0);
            words(1, w1);
            words(2, w2);
            fill(0, w0);
            cp_async_commit();
            fill(1, w1);
            cp_async_commit();
            for (int b = 0; b < nbt; ++b) {
                cp_async_wait<1>();
                __syncthreads();       // batch b is in; the adder is done with batch b - 1
#pragma unroll
                for (int i = 0; i < NWD; ++i) w0[i] = w2[i];
                words(b + 3, w2);
                fill(b + 2, w0);
                cp_async_commit();
            }
            cp_async_wait<0>();
        } else {
            T acc = T(0);
            for (int b = 0; b < nbt; ++b) {
                __syncthreads();
                const T *x = xs + (b % kHubStages) * (NB * GH) + lg;
                const int n = min(NB, deg - b * NB);
                int i = 0;
                for (; i + 32 <= n; i += 32) {
                    T y[32];
#pragma unroll
                    for (int u = 0; u < 32; ++u) y[u] = x[(i + u) * GH];
#pragma unroll
                    for (int u = 0; u < 32; ++u) acc = add_rn(acc, y[u]);
                }
                for (; i < n; ++i) acc = add_rn(acc, x[i * GH]);
            }
            if (sub == 0 && col0 + lg < a.nA) reinterpret_cast<T *>(a.out)[(size_t)v * a.out_pitch + col0 + lg] = acc;
        }
    }
}

// Wide.  A warp walks the neighbour entries of its vertices as one stream
// through a ring of RR rows in shared memory, BR of them a copy group
// (cp.async, the 16-byte pieces that the neighbour's color needs).  A lane
// then reads, for each of its slots, the element the color points at (a zero
// behind the row where it points at none).  What depends on the color and
// the lane alone (which pieces, which of a slot's sets) is a bit per color in
// registers, tested against 1 << color; the offsets are a table in shared
// memory, eight to a load.
__device__ __forceinline__ float lds_elem(uint32_t addr, float)
{
    float x;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr));
    return x;
}
__device__ __forceinline__ double lds_elem(uint32_t addr, double)
{
    double x;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(addr));
    return x;
}
// base + the low or high half of w, in one instruction
__device__ __forceinline__ uint32_t add_lo(uint32_t base, uint32_t w) { return __dp2a_lo(w, 0x0001u, base); }
__device__ __forceinline__ uint32_t add_hi(uint32_t base, uint32_t w) { return __dp2a_lo(w, 0x0100u, base); }

template <int R> __device__ __forceinline__ void add_all(float (&acc)[R], const float (&x)[R])
{
#pragma unroll
    for (int r = 0; r + 1 < R; r += 2) {
        unsigned long long a, b;
        asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(acc[r]), "f"(acc[r + 1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(x[r]), "f"(x[r + 1]));
        a = add2_rn(a, b);
        asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[r]), "=f"(acc[r + 1]) : "l"(a));
    }
    if (R & 1) acc[R - 1] = add_rn(acc[R - 1], x[R - 1]);
}
template <int R> __device__ __forceinline__ void add_all(double (&acc)[R], const double (&x)[R])
{
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = add_rn(acc[r], x[r]);
}

// a += x where `second` is 0, else b += x
__device__ __forceinline__ void add_one_of(float &a, float &b, float x, uint32_t second)
{
    asm("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %3, 0;\n\t@p add.rn.f32 %0, %0, %2;\n\t@!p add.rn.f32 %1, %1, %2;\n\t}"
        : "+f"(a), "+f"(b)
        : "f"(x), "r"(second));
}
__device__ __forceinline__ void add_one_of(double &a, double &b, double x, uint32_t second)
{
    asm("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %3, 0;\n\t@p add.rn.f64 %0, %0, %2;\n\t@!p add.rn.f64 %1, %1, %2;\n\t}"
        : "+d"(a), "+d"(b)
        : "d"(x), "r"(second));
}
__device__ __forceinline__ void add_if(float &a, float x, uint32_t on)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p add.rn.f32 %0, %0, %1;\n\t}" : "+f"(a) : "f"(x), "r"(on));
}
__device__ __forceinline__ void add_if(double &a, double x, uint32_t on)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p add.rn.f64 %0, %0, %1;\n\t}" : "+d"(a) : "d"(x), "r"(on));
}

// bytes between the ring's rows: the row and a zero, in whole lines as the table's rows
__host__ __device__ inline uint32_t wide_stride(uint32_t row_bytes) { return (row_bytes + 16u + 127u) / 128u * 128u; }

template <int R> constexpr int wide_ids() { return R <= 8 ? 8 : 16; }

template <typename T, int R, int M, int RR, int BR, int NP>
__global__ void __launch_bounds__(kGatherThreads) k_gather_wide(GatherArgs a)
{
    constexpr int N = wide_ids<R>(), NC = N / 8, PF = RR - BR;   // PF: rows copied ahead
    constexpr int PE = 16 / (int)sizeof(T);
    constexpr int MB = M == 1 ? 0 : M == 2 ? 1 : M;              // member masks a slot (two members: the second's)
    static_assert(32 % RR == 0 && RR % BR == 0 && PF % BR == 0 && PF > 0, "a ring divides 32 entries");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t need[NP][32], member[MB ? MB * R : 1][32];   // [..][lane]: a bit per color
    // [k][N / 8][32][8] byte offsets in a row slot; color 0: the zero behind the row
    uint16_t *tab = reinterpret_cast<uint16_t *>(smem_raw);
    unsigned char *ring_raw = smem_raw + (size_t)a.k * 32 * N * 2;   // a multiple of 512 bytes
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t row_bytes = ((uint32_t)a.nR * (uint32_t)sizeof(T) + 15u) / 16u * 16u, rs = wide_stride(row_bytes);
    const int slot0 = blockIdx.y * (32 * R);
    __shared__ int s_turn;
    if (threadIdx.x == 0 && blockIdx.y == 0) s_turn = hub_turn(a);
    for (int i = threadIdx.x; i < NP * 32; i += kGatherThreads) (&need[0][0])[i] = 0;
    for (int i = threadIdx.x; i < MB * R * 32; i += kGatherThreads) (&member[0][0])[i] = 0;
    __syncthreads();
    // four entries a thread at a time, their loads in flight together: on a graph of
    // a hundred vertices the tables are the kernel's time
    for (int i0 = threadIdx.x; i0 < a.k * 32 * N; i0 += 4 * kGatherThreads) {
        uint16_t y[4][M];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kGatherThreads, d = i / (32 * N), l = i / 8 % 32, r = i / 256 % NC * 8 + i % 8;
            const int slot = slot0 + r * 32 + l;
#pragma unroll
            for (int m = 0; m < M; ++m)
                y[u][m] = d > 0 && d < a.k && r < R && slot < a.start[m + 1] - a.start[m]
                              ? __ldg(a.idx + (size_t)(d - 1) * a.nA + a.start[m] + slot)
                              : (uint16_t)0xffffu;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kGatherThreads;
            if (i >= a.k * 32 * N) break;
            const int d = i / (32 * N), l = i / 8 % 32, r = i / 256 % NC * 8 + i % 8;
            uint16_t x = 0xffffu;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                if (y[u][m] == 0xffffu) continue;
                x = y[u][m];
                if (MB == 1 && m == 1) atomicOr(&member[r][l], 1u << d);
                if (MB > 1) atomicOr(&member[r * MB + m][l], 1u << d);
            }
            if (x != 0xffffu) {   // whole sectors: the two pieces of 32 bytes
                const int q = x / PE & ~1;
                atomicOr(&need[q >> 5][q & 31], 1u << d);
                if ((uint32_t)(q + 1) * 16 < row_bytes) atomicOr(&need[q >> 5][(q & 31) + 1], 1u << d);
            }
            tab[i] = (uint16_t)(x == 0xffffu ? row_bytes : (uint32_t)x * (uint32_t)sizeof(T));
        }
    }
    if (blockIdx.y == 0 && s_turn) hub_part<T, 32>(a, ring_raw);
    __syncthreads();
    for (int i = threadIdx.x; i < kWarps * RR; i += kGatherThreads)
        *reinterpret_cast<uint4 *>(ring_raw + (size_t)i * rs + row_bytes) = make_uint4(0, 0, 0, 0);
    uint32_t nd[NP], mb[MB ? MB * R : 1];
#pragma unroll
    for (int p = 0; p < NP; ++p) nd[p] = need[p][lane];
#pragma unroll
    for (int i = 0; i < MB * R; ++i) mb[i] = member[i][lane];
    __syncthreads();
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(ring_raw) + (uint32_t)(warp * RR) * rs;
    const char *aux = reinterpret_cast<const char *>(a.aux) + lane * 16;
    const uint32_t pitch_bytes = (uint32_t)a.pitch * (uint32_t)sizeof(T);
    const uint16_t *mytab = tab + lane * 8;
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(a.ticket + blockIdx.y, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        int v0, v1;
        if (!chunk_of(a.map, t, v0, v1)) break;
        const int e0 = __ldg(a.off + v0), ends = __ldg(a.off + min(v0 + 1 + lane, v1)) - e0;   // a chunk has at most 32 vertices
        const int n = __shfl_sync(0xffffffffu, ends, v1 - v0 - 1);
        auto word = [&](int g) { return g * 32 + lane < n ? (uint32_t)__ldg(a.adjd + e0 + g * 32 + lane) : 0u; };
        // the words of 32 entries (wA), of the next 32 (wB) and of those after
        uint32_t wA = word(0), wB = word(1), wC = word(2);
        uint32_t color[RR];   // of the ring's rows
        auto issue = [&](int rr, uint32_t w, int from) {
            const uint32_t x = __shfl_sync(0xffffffffu, w, from);
            color[rr] = x >> 28;
            const uint32_t bit = 1u << (x >> 28);
            const char *src = aux + (uint64_t)(x & 0x0fffffffu) * pitch_bytes;
            const uint32_t dst = ring + (uint32_t)rr * rs + (uint32_t)lane * 16u;
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (nd[p] & bit) cp_async16_s(dst + p * 512, src + p * 512);
        };
        T acc[M][R];
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[m][r] = T(0);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < PF; ++q) {
            issue(q, wA, q);
            if (q % BR == BR - 1) cp_async_commit();
        }
        int v = v0, vend = __shfl_sync(0xffffffffu, ends, 0);
        for (int b = 0; b < n; b += RR) {
            const int at = b & 31;                       // in wA
            const uint32_t wN = at + RR == 32 ? wB : wA; // of the entries RR further
#pragma unroll
            for (int q = 0; q < RR; q += BR) {
                if (b + q >= n) break;
#pragma unroll
                for (int i = 0; i < BR; ++i) {
                    const int f = q + PF + i;
                    issue(f % RR, f < RR ? wA : wN, (at + f) & 31);
                }
                cp_async_commit();
                cp_async_wait<PF / BR>();
                __syncwarp();
                uint4 id[BR][NC];
#pragma unroll
                for (int i = 0; i < BR; ++i)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        id[i][c] = *reinterpret_cast<const uint4 *>(mytab + (color[q + i] * NC + c) * 256);
#pragma unroll
                for (int i = 0; i < BR; ++i) {
                    const uint32_t row = ring + (uint32_t)(q + i) * rs, bit = 1u << color[q + i];
                    T x[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const uint4 z = id[i][r / 8];
                        const uint32_t w = (r & 7) < 2 ? z.x : (r & 7) < 4 ? z.y : (r & 7) < 6 ? z.z : z.w;
                        x[r] = lds_elem(r & 1 ? add_hi(row, w) : add_lo(row, w), T(0));
                    }
                    if constexpr (M == 1) {
                        add_all<R>(acc[0], x);
                    } else {
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            if constexpr (M == 2) {
                                add_one_of(acc[0][r], acc[1][r], x[r], mb[r] & bit);
                            } else {
#pragma unroll
                                for (int m = 0; m < M; ++m) add_if(acc[m][r], x[r], mb[r * MB + m] & bit);
                            }
                        }
                    }
                    if (b + q + i + 1 == vend) {
                        T *o = reinterpret_cast<T *>(a.out) + (size_t)v * a.out_pitch + slot0 + lane;
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            const int cols = a.start[m + 1] - a.start[m] - slot0 - lane;
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                if (r * 32 < cols) o[a.start[m] + r * 32] = acc[m][r];
                                acc[m][r] = T(0);
                            }
                        }
                        ++v;
                        vend = __shfl_sync(0xffffffffu, ends, (v - v0) & 31);
                    }
                }
                __syncwarp();
            }
            if (at + RR == 32) {
                wA = wB;
                wB = wC;
                wC = word((b >> 5) + 3);
            }
        }
        cp_async_wait<0>();
    }
}

// Narrow.  U neighbours in flight a lane, their words loaded once a group of
// G lanes (a batch ahead) and passed round by shuffles.  A slot of which no set
// holds the neighbour's color loads nothing: a bit per color and slot in a
// register, as for which of two sets it is; with more sets a slot the member
// is in the table's entry (above the column's 13 bits) and the sums are in
// shared memory.  The warp's vertices (of like degree) take as many batches as
// the longest list of them.
template <int R> struct Ids { static constexpr int n = R <= 1 ? 1 : R <= 2 ? 2 : R <= 4 ? 4 : R <= 8 ? 8 : 16; };

template <int N> __device__ __forceinline__ void load_ids(const uint16_t *p, uint32_t (&w)[(N + 1) / 2])
{
    if constexpr (N == 1) {
        w[0] = *p;
    } else if constexpr (N == 2) {
        w[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (N == 4) {
        const uint2 t = *reinterpret_cast<const uint2 *>(p);
        w[0] = t.x; w[1] = t.y;
    } else {
#pragma unroll
        for (int i = 0; i < N / 8; ++i) {
            const uint4 t = *(reinterpret_cast<const uint4 *>(p) + i);
            w[4 * i] = t.x; w[4 * i + 1] = t.y; w[4 * i + 2] = t.z; w[4 * i + 3] = t.w;
        }
    }
}

__device__ __forceinline__ float ld_if(const float *p, uint32_t on)
{
    float x;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
        : "=f"(x)
        : "l"(p), "r"(on));
    return x;
}
__device__ __forceinline__ double ld_if(const double *p, uint32_t on)
{
    double x;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t@q ld.global.nc.f64 %0, [%1];\n\t}"
        : "=d"(x)
        : "l"(p), "r"(on));
    return x;
}

template <typename T, int G, int R, int M, int U, int GH> __global__ void __launch_bounds__(kGatherThreads) k_gather(GatherArgs a)
{
    constexpr int N = Ids<R>::n, WPL = (U + G - 1) / G;   // WPL: words a lane loads of a batch
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t hits[R][G], seconds[R][G];            // a bit per color: some set holds it; the second does
    uint16_t *tab = reinterpret_cast<uint16_t *>(smem_raw);   // [k][G][N]
    const int slot0 = blockIdx.y * (G * R);
    __shared__ int s_turn;
    if (threadIdx.x == 0 && blockIdx.y == 0) s_turn = hub_turn(a);
    for (int i = threadIdx.x; i < R * G; i += kGatherThreads) (&hits[0][0])[i] = (&seconds[0][0])[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < a.k * G * N; i += kGatherThreads) {
        const int d = i / (G * N), l = (i - d * (G * N)) / N, r = i % N;
        const int slot = slot0 + r * G + l;
        uint16_t x = 0;
        if (d > 0 && r < R)
            for (int m = 0; m < M; ++m) {
                if (slot >= a.start[m + 1] - a.start[m]) break;
                const uint16_t y = __ldg(a.idx + (size_t)(d - 1) * a.nA + a.start[m] + slot);
                if (y == 0xffffu) continue;
                x = (uint16_t)(M > 2 ? y | m << 13 : y);
                atomicOr(&hits[r][l], 1u << d);
                if (m == 1) atomicOr(&seconds[r][l], 1u << d);
            }
        tab[i] = x;
    }
    unsigned char *rest = smem_raw + ((size_t)a.k * G * N * 2 + 15) / 16 * 16;
    if (blockIdx.y == 0 && s_turn) hub_part<T, GH>(a, rest);
    __syncthreads();
    T *sacc = reinterpret_cast<T *>(rest) + threadIdx.x;   // M > 2: [R][M][threads], a thread's own
    const int lane = threadIdx.x & 31, lg = lane % G, grp = lane / G;
    uint32_t hit[R], second[R];
#pragma unroll
    for (int r = 0; r < R; ++r) hit[r] = hits[r][lg], second[r] = seconds[r][lg];
    const uint16_t *mytab = tab + lg * N;
    const T *aux = reinterpret_cast<const T *>(a.aux);
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(a.ticket + blockIdx.y, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        int v0, v1;
        if (!chunk_of(a.map, t, v0, v1)) break;
        if constexpr (R == 1 && G <= 4) {
            // long lists of few slots: a warp a vertex, the groups of G lanes each
            // fetch a neighbour, DEP batches ahead, and every group adds all of them in
            // order (by shuffles).  Eight vertices a warp left lists of 3000 neighbours
            // with eight in flight: 0.29 ms at 12 M entries and four slots, now 0.18.
            // At eight slots of three sets the adds cost more than the wait (0.9 ->
            // 1.2 ms at 31 M entries).
            if (__ldg(a.off + v0 + 1) - __ldg(a.off + v0) >= (G == 1 ? 32 : 128)) {
                constexpr int NPF = 32 / G, DEP = G == 1 ? 3 : 6;
                for (int v = v0; v < v1; ++v) {
                    const int beg = __ldg(a.off + v), end = __ldg(a.off + v + 1);
                    auto word = [&](int e) { return e + grp < end ? (uint32_t)__ldg(a.adjd + e + grp) : 0u; };
                    T x[DEP], acc[M];
                    uint32_t mem[DEP], z[DEP];
                    auto fetch = [&](int q, uint32_t y) {
                        const uint32_t bit = 1u << (y >> 28), c = mytab[(y >> 28) * G];
                        x[q] = ld_if(aux + (size_t)(y & 0x0fffffffu) * (uint32_t)a.pitch + (M > 2 ? c & 0x1fffu : c), hit[0] & bit);
                        mem[q] = M > 2 ? c >> 13 : second[0] & bit;
                    };
#pragma unroll
                    for (int m = 0; m < M; ++m) acc[m] = T(0);
#pragma unroll
                    for (int q = 0; q < DEP; ++q) z[q] = word(beg + q * NPF);
#pragma unroll
                    for (int q = 0; q < DEP; ++q) {
                        fetch(q, z[q]);
                        z[q] = word(beg + (DEP + q) * NPF);
                    }
                    for (int e = beg; e < end; e += DEP * NPF) {
#pragma unroll
                        for (int q = 0; q < DEP; ++q) {
                            if (e + q * NPF >= end) break;
#pragma unroll
                            for (int i = 0; i < NPF; ++i) {
                                const T y = __shfl_sync(0xffffffffu, x[q], i * G + lg);
                                if constexpr (M == 1) {
                                    acc[0] = add_rn(acc[0], y);
                                } else {
                                    const uint32_t who = __shfl_sync(0xffffffffu, mem[q], i * G + lg);
                                    if constexpr (M == 2) {
                                        add_one_of(acc[0], acc[1], y, who);
                                    } else {
#pragma unroll
                                        for (int m = 0; m < M; ++m) add_if(acc[m], y, who == (uint32_t)m);
                                    }
                                }
                            }
                            fetch(q, z[q]);
                            z[q] = word(e + (2 * DEP + q) * NPF);
                        }
                    }
                    if (grp == 0) {
#pragma unroll
                        for (int m = 0; m < M; ++m)
                            if (slot0 + lg < a.start[m + 1] - a.start[m])
                                reinterpret_cast<T *>(a.out)[(size_t)v * a.out_pitch + slot0 + a.start[m] + lg] = acc[m];
                    }
                }
                continue;
            }
        }
        for (int vb = v0; vb < v1; vb += 32 / G) {
            const int v = vb + grp;
            T acc[M][R];
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[m][r] = T(0);
                    if (M > 2) sacc[(r * M + m) * kGatherThreads] = T(0);
                }
            const int beg = v < v1 ? __ldg(a.off + v) : 0, end = v < v1 ? __ldg(a.off + v + 1) : 0;
            const int most = __reduce_max_sync(0xffffffffu, end - beg);
            uint32_t w[WPL];
            auto words = [&](int e) {
#pragma unroll
                for (int i = 0; i < WPL; ++i)
                    w[i] = i * G + lg < U && e + i * G + lg < end ? (uint32_t)__ldg(a.adjd + e + i * G + lg) : 0u;
            };
            words(beg);
            for (int b = 0; b < most; b += U) {
                T x[U][R];
                uint32_t mem[U][R];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t z = G == 1 ? w[u % WPL] : __shfl_sync(0xffffffffu, w[u / G], lane - lg + u % G);
                    const uint32_t bit = 1u << (z >> 28);
                    uint32_t id[(N + 1) / 2];
                    load_ids<N>(mytab + (z >> 28) * (G * N), id);
                    const T *row = aux + (size_t)(z & 0x0fffffffu) * (uint32_t)a.pitch;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const uint32_t c = N == 1 ? id[0] : r & 1 ? id[r / 2] >> 16 : id[r / 2] & 0xffffu;
                        x[u][r] = ld_if(row + (M > 2 ? c & 0x1fffu : c), hit[r] & bit);
                        mem[u][r] = M > 2 ? c >> 13 : second[r] & bit;
                    }
                }
                words(beg + b + U);
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if constexpr (M == 1) {
                            acc[0][r] = add_rn(acc[0][r], x[u][r]);
                        } else if constexpr (M == 2) {
                            add_one_of(acc[0][r], acc[1][r], x[u][r], mem[u][r]);
                        } else {
                            T *p = sacc + (r * M + mem[u][r]) * kGatherThreads;
                            *p = add_rn(*p, x[u][r]);
                        }
                    }
            }
            if (v >= v1) continue;
            T *o = reinterpret_cast<T *>(a.out) + (size_t)v * a.out_pitch + slot0;
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (slot0 + r * G + lg < a.start[m + 1] - a.start[m])
                        o[a.start[m] + r * G + lg] = M > 2 ? sacc[(r * M + m) * kGatherThreads] : acc[m][r];
        }
    }
}

namespace {

int gather_grid(const GatherArgs &a, int per_sm, int sm_count, int hub_cols)
{
    const int64_t items = (int64_t)a.hubs * ((a.nA + hub_cols - 1) / hub_cols);
    const int64_t want = (a.map.base[a.map.n] + kWarps - 1) / kWarps + items;
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)sm_count * per_sm, want));
}

template <typename T, int G, int R, int M, int U, int GH> void go_narrow_h(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    const size_t sacc = M > 2 ? (size_t)R * M * kGatherThreads * sizeof(T) : 0;
    const size_t smem = ((size_t)a.k * G * Ids<R>::n * 2 + 15) / 16 * 16 + std::max(sacc, a.hubs > 0 ? hub_bytes<T, GH>() : 0);
    auto kern = k_gather<T, G, R, M, U, GH>;
    const int per_sm = resident_ctas((const void *)kern, kGatherThreads, smem);
    kern<<<dim3(gather_grid(a, per_sm, sm_count, GH), (a.slots + G * R - 1) / (G * R)), kGatherThreads, smem, st>>>(a);
}

template <typename T, int G, int R, int M, int U> void go_narrow(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    if constexpr (G * R * M == 1) return go_narrow_h<T, G, R, M, U, 1>(a, sm_count, st);
    if constexpr (G * R * M <= 8) return go_narrow_h<T, G, R, M, U, 8>(a, sm_count, st);
    if (a.nA <= 8) return go_narrow_h<T, G, R, M, U, 8>(a, sm_count, st);
    if (a.nA <= 16) return go_narrow_h<T, G, R, M, U, 16>(a, sm_count, st);
    return go_narrow_h<T, G, R, M, U, 32>(a, sm_count, st);
}

template <typename T, int M> void pick_narrow(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    const int n = a.slots;
    if constexpr (M == 1)
        if (n <= 1) return go_narrow<T, 1, 1, 1, 8>(a, sm_count, st);
    if constexpr (M <= 2)
        if (n <= 4) return go_narrow<T, 4, 1, M, 8>(a, sm_count, st);
    if constexpr (M <= 4)
        if (n <= 8) return go_narrow<T, 8, 1, M, 8>(a, sm_count, st);
    if (n <= 16) return go_narrow<T, 16, 1, M, 8>(a, sm_count, st);
    if (n <= 32) return go_narrow<T, 32, 1, M, 8>(a, sm_count, st);
    if (n <= 64) return go_narrow<T, 32, 2, M, 4>(a, sm_count, st);
    return go_narrow<T, 32, 4, M, 2>(a, sm_count, st);
}

// Rows in the ring.  Eight (sixteen short ones, four of the longest) measured
// fastest: at 131,072 vertices of degree 32 and 12 colors, rows of 1848 bytes
// take 0.82 ms with four and three CTAs an SM, 0.75 with eight and one; rows of
// 1320 bytes 0.71 with sixteen and one CTA, 0.55 with eight and two.
constexpr size_t kWideSmem = 215 * 1024;
inline int wide_ring(size_t row_bytes) { return row_bytes <= 512 ? 16 : row_bytes <= 2816 ? 8 : 4; }
template <typename T> size_t wide_smem(const GatherArgs &a, int ids)
{
    const size_t rb = ((size_t)a.nR * sizeof(T) + 15) / 16 * 16;
    return (size_t)a.k * 32 * ids * 2 +
           std::max((size_t)kWarps * wide_ring(rb) * wide_stride((uint32_t)rb), a.hubs > 0 ? hub_bytes<T, 32>() : 0);
}

template <typename T, int R, int M, int RR, int BR, int NP> void go_wide_n(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    const size_t smem = wide_smem<T>(a, wide_ids<R>());
    auto kern = k_gather_wide<T, R, M, RR, BR, NP>;
    const int per_sm = resident_ctas((const void *)kern, kGatherThreads, smem);
    kern<<<dim3(gather_grid(a, per_sm, sm_count, 32), (a.slots + 32 * R - 1) / (32 * R)), kGatherThreads, smem, st>>>(a);
}

// NP: 16-byte pieces of a row a lane
template <typename T, int R, int M> void go_wide(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    const size_t rb = ((size_t)a.nR * sizeof(T) + 15) / 16 * 16;
    switch (wide_ring(rb)) {
    case 16: return go_wide_n<T, R, M, 16, 4, 1>(a, sm_count, st);
    case 8:
        if (rb <= 1536) return go_wide_n<T, R, M, 8, 4, 3>(a, sm_count, st);
        if (rb <= 2048) return go_wide_n<T, R, M, 8, 2, 4>(a, sm_count, st);
        return go_wide_n<T, R, M, 8, 2, 8>(a, sm_count, st);
    default: return go_wide_n<T, R, M, 4, 2, 8>(a, sm_count, st);
    }
}

template <typename T> bool is_wide(const GatherArgs &a)
{
    return a.slots > 32 && a.nR >= 32 && a.nR * sizeof(T) <= 4096 && wide_smem<T>(a, a.slots <= 256 ? 8 : 16) <= kWideSmem;
}

template <typename T, int M> void pick_wide(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    const int n = a.slots;
    if (n <= 64) return go_wide<T, 2, M>(a, sm_count, st);
    if (n <= 96) return go_wide<T, 3, M>(a, sm_count, st);
    if (n <= 128) return go_wide<T, 4, M>(a, sm_count, st);
    if (n <= 192) return go_wide<T, 6, M>(a, sm_count, st);
    if constexpr (M <= 2) {
        if (n > 256 && n <= 352) return go_wide<T, 11, M>(a, sm_count, st);
        if (n > 256 && n <= 480) return go_wide<T, 15, M>(a, sm_count, st);
    }
    return go_wide<T, 8, M>(a, sm_count, st);
}

template <typename T, int M> void pick_gather(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    if (is_wide<T>(a)) pick_wide<T, M>(a, sm_count, st);
    else pick_narrow<T, M>(a, sm_count, st);
}

template <typename T> void launch_gather_t(const GatherArgs &a, int sm_count, cudaStream_t st)
{
    switch (a.members) {
    case 1: return pick_gather<T, 1>(a, sm_count, st);
    case 2: return pick_gather<T, 2>(a, sm_count, st);
    case 3: return pick_gather<T, 3>(a, sm_count, st);
    case 4: return pick_gather<T, 4>(a, sm_count, st);
    default: return pick_gather<T, 5>(a, sm_count, st);
    }
}

}  // namespace

}  // namespace rt
}  // namespace sg
