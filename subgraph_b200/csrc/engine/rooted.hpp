// Rooted rows: the plain form's tables and steps.
//
// Every colorful embedding rooted at a vertex v uses v's color, so v's row of
// a sub-template of m vertices is non-zero only at the C(k-1, m-1) color sets
// holding color(v).  A rooted row keeps those alone, addressed in the colors
// relative to v's: color x is x - color(v) mod k, v's own color is 0, and the
// set {color(v)} + T is a column for each (m-1)-subset T of the relative colors
// 1 .. k-1 (columns()).  An aggregate over v's neighbours is wanted only at the
// sets without v's color: the m-subsets S of the relative colors 1 .. k-1.
// A neighbour whose relative color is d adds to the sets S holding d, from
// its own row's column {s - d mod k : s in S, s != d}: a table that depends on
// d alone, k - 1 rows of C(k-1, m) columns, serves every pair of vertices.
//
// Columns are ordered in slots: up to kMaxMembers sets without a common color
// share a slot, and a neighbour's color lies in at most one of them, so one
// load serves the whole slot; the first sets of all slots come first, then the
// second ones, and so on, which keeps a warp's columns contiguous.
//
// What is left out are exact zeros (a vertex's sets without its color, the
// neighbours of the vertex's own color) and columns that meet a main entry
// that is an exact zero (aggregate sets holding the vertex's color); the sums
// that remain are in the reference's order: neighbours in list order
// (CSCGraph.hpp:242-307), splits in lex order of the colors themselves
// (DataTableColMajor.cpp:346-500).
//
// Vertices whose rows nobody reads are left out too.  Internal ids descend in
// degree: a vertex without neighbours has only zero rows, and the row of a
// vertex with one neighbour u holds u's color in every non-zero set, so it
// adds nothing to u (its only reader) and nothing to its own larger
// sub-templates, whose next neighbour would be u again.  Tables therefore
// have the V2 rows of the vertices of degree 2 or more; only the root step
// also reads the vertices of degree 1 (V1).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../host/plan.hpp"
#include "stage.cuh"

namespace sg {
namespace rt {

// Vertices in chunks for the kernels' tickets: class c holds the vertices
// [first[c], first[c + 1]) of the degree-descending order, per[c] of them a
// chunk, chunk ids from base[c].
constexpr int kMaxClass = 26;
struct ChunkMap {
    int32_t n;                          // classes
    int32_t first[kMaxClass + 1];
    int32_t base[kMaxClass + 1];        // base[n]: chunks in all
    int32_t per[kMaxClass];
};

constexpr int kMaxMembers = 5;
struct ColumnOrder {
    std::vector<unsigned> sets;         // bit i: relative color i + 1
    std::vector<int> pos;               // column of a set
    int members = 1, slots = 0;
    int start[kMaxMembers + 1];         // the m-th sets of the slots: columns [start[m], start[m + 1])
};
// the columns of the `size`-subsets of k - 1 relative colors
const ColumnOrder &columns(int k, int size);

struct EdgeArgs {
    int32_t V1, lim, k;                 // rows of vertices [0, V1); neighbours at or past lim are not gathered
    int32_t hubs;                       // vertices [0, hubs): one CTA each
    const int32_t *off, *adj;
    const uint8_t *color;
    int32_t *adjd;                      // [nnz] neighbour | its relative color << 28 (0: adds nothing), or null
    void *cnt, *scnt;                   // [V1][cnt_pitch] neighbours of each relative color; the same scaled, or null
    int32_t cnt_pitch;
};

struct GatherArgs {
    int32_t k, nA, nR, V;               // aggregate columns, row columns, vertices [0, V)
    int32_t pitch, out_pitch;           // of the gathered rows and of the result (elements)
    int32_t hubs;                       // vertices [0, hubs): the CTA-wide part
    const int32_t *off, *adjd;
    const void *aux;
    void *out;
    int32_t members, slots, start[kMaxMembers + 1];   // of the aggregate's columns (ColumnOrder)
    const uint16_t *idx;                // [k-1][nA] column of the neighbour's row, 0xffff: adds nothing
    ChunkMap map;                       // of the vertices [hubs, V)
    int32_t *ticket, *hub_ticket;       // zeroed: a chunk counter per column block; the hub items' counter
    uint32_t *sm_seen;                  // zeroed: a bit per SM that has a CTA [kSmWords]
    int32_t spread;                     // hub items: one CTA of an SM takes them
};
// counters of a step: column blocks (at most kColumnBlocks), SMs, hub items
constexpr int kColumnBlocks = 56, kSmWords = 7, kStepTickets = kColumnBlocks + kSmWords + 1;

struct EmaArgs {
    int32_t k, V, nA, nM, nO, S;        // columns of aggregate, main and result rows; splits per result
    int32_t agg_pitch, main_pitch, out_pitch;
    int32_t tile_v, is_root, fused;     // fused: multiply-adds with one rounding (the split loop)
    const void *agg, *main;
    void *out;
    const uint8_t *color;
    // rank of each relative column in the order of the colors themselves
    // without the vertex's own: [k][columns]
    const uint16_t *perm_a, *perm_m, *perm_o;
    const uint32_t *split;              // [S][split_stride] main rank | aggregate rank << 16
    int32_t split_stride;
    const int32_t *blk;                 // block tables (blk_sched.hpp), or null: the split loop
    int32_t blk_shape, blk_nblocks;
    double *root_value;                 // root: per vertex
};

struct RootArgs {
    int32_t V1, pitch, tile_v;
    const void *val;                    // [V1][pitch] root values: the aggregate (one-hot main), or doubles
    double *root_partial, *root_vertex; // per tile, per vertex (optional)
};

// vertices [hubs, mid) a warp each, [mid, low) 8 threads each, [low, V1) 2
void launch_edges(const EdgeArgs &a, int32_t mid, int32_t low, bool fp64, cudaStream_t st);
// false: the shapes do not fit the kernels (the caller takes the general path)
bool gather_fits(int k, int nA, int nR, bool fp64);
int gather_lanes(const GatherArgs &a);  // threads a vertex
void launch_gather_f32(const GatherArgs &a, int sm_count, cudaStream_t st);
void launch_gather_f64(const GatherArgs &a, int sm_count, cudaStream_t st);
// returns the kernels launched
int launch_gather(const GatherArgs &a, bool fp64, int sm_count, cudaStream_t st);
int ema_tile(int nA, int nM, int nO, bool fp64, bool root, bool blocked);   // vertices a tile, 0: does not fit
void launch_ema(const EmaArgs &a, bool fp64, cudaStream_t st);
int launch_root_tiles(const RootArgs &a, bool fp64, cudaStream_t st);   // returns the tiles (= partials)

// ---- host plan -------------------------------------------------------------
// One step of process_order: the sub's table is an alias of the neighbour
// counts (two vertices), a gather, or a gather (or the counts) and a product.
struct Step {
    int s = 0;
    bool main_leaf = false, aux_leaf = false;
    int m = 0, pm = 0, n = 0;           // vertices of the aux child, the main child, the sub
    int nA = 0, nM = 0, nO = 0;
    int root_tile = 32;                 // root: vertices a tile of its sum
    bool fused = false;                 // outside exact mode: multiply-adds with one rounding
};
struct SubTable {
    int kind = 0;                       // 0 none, 1 the counts, 2 the scaled counts, 3 the arena
    int pitch = 0;
    int64_t off = -1;                   // arena units (elements a vertex)
};
struct RootedPlan {
    bool ok = false;
    int k = 0, cnt_pitch = 0, agg_pitch = 0;
    bool need_edges = false, need_scaled = false;
    std::vector<Step> steps;
    std::vector<SubTable> tab;          // per sub
    int64_t arena_units = 0;
};
RootedPlan make_rooted_plan(const Plan &p, bool fp64);

// Device tables of a plan (they depend on the template alone).
struct RootedTables {
    void *mem = nullptr;                // one allocation
    std::vector<const uint16_t *> idx;  // per step
    std::vector<const uint16_t *> perm; // per subset size: [k][C(k-1, size)]
    std::vector<const uint32_t *> split;
    std::vector<int32_t> split_stride, S;
    std::vector<const int32_t *> blk;
    std::vector<int32_t> blk_shape, blk_nblocks;
};
// Builds the tables of a plan and copies them to the device, in memory of the
// device's pool (a template made and dropped per call paid 0.4 ms and more for
// the driver's own allocation).
cudaError_t upload_rooted_tables(const Plan &p, const RootedPlan &rp, RootedTables &t, cudaStream_t st);

// blocks of an index structure (engine.cu): the register-blocked schedule
bool rooted_blocks(int k, int n, int pm, std::vector<int32_t> &rows, int &nblocks, int &shape);

// chunks of about `target` entries, at least `least` vertices each (one where a
// vertex has `alone` neighbours or more, a power of two), at most `most`
ChunkMap make_chunks(const std::vector<int32_t> &degree, int32_t first, int32_t last, int target, int least, int alone,
                     int most);

}  // namespace rt
}  // namespace sg
