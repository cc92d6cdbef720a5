// Host side of the rooted rows (rooted.hpp): the steps of a template, the
// layout of its tables and the index tables the kernels read.
#include "rooted.hpp"

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>

namespace sg {
namespace rt {

namespace {

int round_to(int x, int m) { return (x + m - 1) / m * m; }

// Row pitch of a rooted table: 16 bytes for the narrowest rows, whole 32-byte
// sectors, whole 128-byte lines from one line on.  A copy to shared memory
// whose source and destination differ modulo 128 bytes fetches sectors twice
// (measured: 1.27 to 1.87 times the row's sectors).
int row_pitch(int cols, bool fp64)
{
    if (fp64) return round_to(cols, cols <= 2 ? 2 : cols < 16 ? 4 : 16);
    return round_to(cols, cols <= 4 ? 4 : cols < 32 ? 8 : 32);
}

int rank_of(unsigned mask)
{
    int c[32], n = 0;
    for (int b = 0; b < 32; ++b)
        if (mask >> b & 1u) c[n++] = b;
    return colex_rank(c, n);
}

}  // namespace

const ColumnOrder &columns(int k, int size)
{
    static std::mutex mu;
    static std::map<std::pair<int, int>, ColumnOrder> orders;
    std::lock_guard<std::mutex> lk(mu);
    auto it = orders.find({k, size});
    if (it != orders.end()) return it->second;
    const int n = k - 1;
    std::vector<unsigned> all;
    for (unsigned m = 0; m < (1u << n); ++m)
        if (__builtin_popcount(m) == size) all.push_back(m);
    ColumnOrder o;
    o.members = size < 2 ? 1 : std::min(kMaxMembers, n / size);
    std::vector<std::vector<unsigned>> slots;
    if (o.members == 1) {
        for (unsigned m : all) slots.push_back({m});
    } else {
        // greedy: the next set in colex order, then each time the disjoint set
        // with the fewest disjoint sets left, so that few sets stay alone
        std::vector<int> partners(all.size(), 0);
        std::vector<char> used(all.size(), 0);
        for (size_t a = 0; a < all.size(); ++a)
            for (size_t b = 0; b < all.size(); ++b) partners[a] += (all[a] & all[b]) == 0;
        auto take = [&](size_t a) {
            used[a] = 1;
            for (size_t b = 0; b < all.size(); ++b) partners[b] -= (all[a] & all[b]) == 0;
        };
        for (size_t a = 0; a < all.size(); ++a) {
            if (used[a]) continue;
            take(a);
            std::vector<unsigned> g{all[a]};
            unsigned u = all[a];
            while ((int)g.size() < o.members) {
                int best = -1;
                for (size_t b = 0; b < all.size(); ++b)
                    if (!used[b] && !(all[b] & u) && (best < 0 || partners[b] <= partners[best])) best = (int)b;
                if (best < 0) break;
                take((size_t)best);
                g.push_back(all[best]);
                u |= all[best];
            }
            slots.push_back(g);
        }
        std::stable_sort(slots.begin(), slots.end(), [](auto &a, auto &b) { return a.size() > b.size(); });
    }
    o.slots = (int)slots.size();
    o.pos.assign((size_t)1 << n, -1);
    for (int m = 0; m < kMaxMembers; ++m) {
        o.start[m] = (int)o.sets.size();
        for (auto &g : slots)
            if ((int)g.size() > m) {
                o.pos[g[m]] = (int)o.sets.size();
                o.sets.push_back(g[m]);
            }
    }
    o.start[kMaxMembers] = (int)o.sets.size();
    return orders.emplace(std::make_pair(k, size), std::move(o)).first->second;
}

RootedPlan make_rooted_plan(const Plan &p, bool fp64)
{
    RootedPlan r;
    const int k = p.k, ns = p.nsub();
    r.k = k;
    r.cnt_pitch = row_pitch(k - 1, fp64);
    r.tab.assign(ns, SubTable());
    r.ok = true;
    for (int s : p.process_order) {
        const SubTemplate &st = p.subs[s];
        const SubTemplate &m = p.subs[st.main], &a = p.subs[st.aux];
        if (s != 0) {
            if (p.same_as[s] >= 0) {
                r.tab[s] = r.tab[p.same_as[s]];
                continue;
            }
            SubTable &t = r.tab[s];
            if (m.size == 1 && a.size == 1) {   // the neighbour counts themselves
                t.kind = (!fp64 && s == p.scaled_sub) ? 2 : 1;
                t.pitch = r.cnt_pitch;
                if (t.kind == 2) r.need_scaled = true;
                continue;
            }
            t.kind = 3;
            t.pitch = row_pitch((int)binom(k - 1, st.size - 1), fp64);
        }
        Step q;
        q.s = s;
        q.main_leaf = m.size == 1;
        q.aux_leaf = a.size == 1;
        q.m = a.size;
        q.pm = m.size;
        q.n = st.size;
        q.nA = (int)binom(k - 1, a.size);
        q.nM = q.main_leaf ? 0 : (int)binom(k - 1, m.size - 1);
        q.nO = s == 0 ? 1 : (int)binom(k - 1, st.size - 1);
        if (!q.aux_leaf) {
            const int nR = (int)binom(k - 1, a.size - 1);
            r.need_edges = true;
            r.ok = r.ok && gather_fits(k, q.nA, nR, fp64);
            if (!q.main_leaf || s == 0) r.agg_pitch = std::max(r.agg_pitch, row_pitch(q.nA, fp64));
        }
        if (!q.main_leaf) r.ok = r.ok && ema_tile(q.nA, q.nM, q.nO, fp64, s == 0, false) > 0;
        r.steps.push_back(q);
    }
    // the arena: a table lives from its step to its last reader's
    std::vector<int> readers(ns, 0);
    auto owner = [&](int s) { return p.same_as[s] >= 0 ? p.same_as[s] : s; };
    for (int s : p.process_order)
        if (s != 0) ++readers[owner(s)];
    std::vector<std::pair<int64_t, int64_t>> used;   // (offset, length), sorted
    for (int s : p.process_order) {
        const SubTemplate &st = p.subs[s];
        if (s != 0 && owner(s) == s && r.tab[s].kind == 3) {
            const int64_t len = round_to(r.tab[s].pitch, 32);   // tables start on whole lines
            int64_t at = 0;
            for (auto &u : used) {
                if (at + len <= u.first) break;
                at = std::max(at, u.first + u.second);
            }
            r.tab[s].off = at;
            used.push_back({at, len});
            std::sort(used.begin(), used.end());
            r.arena_units = std::max(r.arena_units, at + len);
        } else if (s != 0 && owner(s) != s) {
            r.tab[s].off = r.tab[owner(s)].off;
        }
        for (int c : {st.main, st.aux})
            if (p.subs[c].size > 1 && --readers[owner(c)] == 0 && r.tab[owner(c)].kind == 3) {
                const int64_t off = r.tab[owner(c)].off;
                used.erase(std::remove_if(used.begin(), used.end(), [&](auto &u) { return u.first == off; }), used.end());
            }
    }
    return r;
}

cudaError_t upload_rooted_tables(const Plan &p, const RootedPlan &rp, RootedTables &t, cudaStream_t st)
{
    const int k = p.k, n = (int)rp.steps.size();
    std::vector<unsigned char> img;
    auto put = [&](const void *src, size_t bytes) -> size_t {
        const size_t at = (img.size() + 255) / 256 * 256;
        img.resize(at + bytes);
        if (bytes) std::memcpy(img.data() + at, src, bytes);
        return at;
    };
    constexpr size_t kNone = ~(size_t)0;
    std::vector<size_t> idx(n, kNone), split(n, kNone), blk(n, kNone), perm(k + 1, kNone);
    std::vector<size_t> idx_m(k + 1, kNone);
    t.split_stride.assign(n, 0);
    t.S.assign(n, 0);
    t.blk_shape.assign(n, 0);
    t.blk_nblocks.assign(n, 0);
    // columns relative to a vertex of color b -> rank in the colors' own order without b
    auto need_perm = [&](int size) {
        if (perm[size] != kNone) return;
        const std::vector<unsigned> &sets = columns(k, size).sets;
        std::vector<uint16_t> v((size_t)k * sets.size());
        for (int b = 0; b < k; ++b)
            for (size_t j = 0; j < sets.size(); ++j) {
                unsigned m = 0;
                for (int i = 0; i < k - 1; ++i)
                    if (sets[j] >> i & 1u) {
                        const int x = (b + i + 1) % k;
                        m |= 1u << (x > b ? x - 1 : x);
                    }
                v[(size_t)b * sets.size() + j] = (uint16_t)rank_of(m);
            }
        perm[size] = put(v.data(), v.size() * 2);
    };
    for (int i = 0; i < n; ++i) {
        const Step &q = rp.steps[i];
        if (!q.aux_leaf) {
            if (idx_m[q.m] == kNone) {
                const std::vector<unsigned> &sets = columns(k, q.m).sets;
                const std::vector<int> &row = columns(k, q.m - 1).pos;
                std::vector<uint16_t> v((size_t)(k - 1) * sets.size(), 0xffffu);
                for (int d = 1; d < k; ++d)
                    for (size_t j = 0; j < sets.size(); ++j) {
                        if (!(sets[j] >> (d - 1) & 1u)) continue;
                        unsigned m = 0;
                        for (int b = 0; b < k - 1; ++b)
                            if ((sets[j] >> b & 1u) && b + 1 != d) m |= 1u << ((b + 1 - d + k) % k - 1);
                        v[(size_t)(d - 1) * sets.size() + j] = (uint16_t)row[m];
                    }
                idx_m[q.m] = put(v.data(), v.size() * 2);
            }
            idx[i] = idx_m[q.m];
        }
        if (q.main_leaf) continue;
        need_perm(q.m);
        need_perm(q.pm - 1);
        if (q.s != 0) need_perm(q.n - 1);
        int L = 0, S = 0;
        std::vector<int32_t> c2c, ms, as;
        index_tables(k - 1, q.n - 1, q.pm - 1, L, S, c2c, ms, as);
        const int stride = round_to(L, 4);
        std::vector<uint32_t> sp((size_t)stride * S, 0u);
        for (int l = 0; l < L; ++l)
            for (int j = 0; j < S; ++j)
                sp[(size_t)j * stride + c2c[l]] =
                    (uint32_t)ms[(size_t)l * S + j] | (uint32_t)as[(size_t)l * S + j] << 16;
        split[i] = put(sp.data(), sp.size() * 4);
        t.split_stride[i] = stride;
        t.S[i] = S;
        std::vector<int32_t> rows;
        if (q.s != 0 && rooted_blocks(k - 1, q.n - 1, q.pm - 1, rows, t.blk_nblocks[i], t.blk_shape[i]))
            blk[i] = put(rows.data(), rows.size() * 4);
    }
    cudaError_t e = cudaMallocAsync(&t.mem, std::max<size_t>(img.size(), 16), st);
    if (e != cudaSuccess) return e;
    if (!img.empty()) {
        // pageable source: the call returns once it has been read
        e = cudaMemcpyAsync(t.mem, img.data(), img.size(), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
    }
    const char *base = (const char *)t.mem;
    auto at = [&](size_t o) { return o == kNone ? nullptr : (const void *)(base + o); };
    for (int i = 0; i < n; ++i) {
        t.idx.push_back((const uint16_t *)at(idx[i]));
        t.split.push_back((const uint32_t *)at(split[i]));
        t.blk.push_back((const int32_t *)at(blk[i]));
    }
    for (int s = 0; s <= k; ++s) t.perm.push_back((const uint16_t *)at(perm[s]));
    return cudaSuccess;
}

ChunkMap make_chunks(const std::vector<int32_t> &degree, int32_t first, int32_t last, int target, int least, int alone,
                     int most)
{
    ChunkMap m{};
    int32_t v = first;
    while (v < last && m.n < kMaxClass) {
        int c = 0;
        while ((2 << c) <= degree[v] && c < 30) ++c;
        // the vertices of degree >= 2^c follow one another
        const int32_t lo = m.n == kMaxClass - 1 ? 0 : (1 << c);
        const int32_t end =
            (int32_t)(std::partition_point(degree.begin() + v, degree.begin() + last, [&](int32_t d) { return d >= lo; }) -
                      degree.begin());
        m.first[m.n] = v;
        m.per[m.n] = std::min(most, std::max((1 << c) >= alone ? 1 : least, target >> c));
        m.base[m.n + 1] = m.base[m.n] + (end - v + m.per[m.n] - 1) / m.per[m.n];
        ++m.n;
        m.first[m.n] = end;
        v = end;
    }
    return m;
}

}  // namespace rt
}  // namespace sg
