"""The work a user has this framework do, as measurable cases.

Every case counts tree templates by color coding on a graph that is resident
on the GPU (or, in the `upload` form, handed over as host arrays), through the
package's public entry points.  The graphs are fixed data sets (seeded R-MAT
graphs of the benchmark's sizes, and uniform random graphs); a case's seed
renames the vertices at random and chooses the colorings, so two seeds give
the same kind of graph with other neighbour lists, colors and counts.

A case: `graph` (rmat, uniform), `V` (any number), `ef` (undirected edges drawn
per vertex), `template` (a name, or the vertices and seed of a random tree),
`n` colorings a pass, `form` (plain, groups, jobs, upload, countmat) and
`mode` (fp32: the reference's arithmetic; exact: without fused products;
fp64: double tables).
"""
import ctypes
import math
import random

import numpy as np
import torch

import subgraph_b200 as sg

# the templates of the benchmark's workloads
TEMPLATES = {
    "p3": (3, [(0, 1), (1, 2)]),
    "tree5": (5, [(0, 1), (1, 2), (2, 3), (1, 4)]),
    "spider7": (7, [(0, 1), (1, 2), (0, 3), (3, 4), (0, 5), (5, 6)]),
    "tree12": (12, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (5, 6), (6, 7), (2, 8), (4, 9), (5, 10), (10, 11)]),
}


def _case(name, graph, V, ef, template, n, form="plain", mode="fp32", tree_n=0, tree_seed=0, jobs=0):
    return {"name": name, "graph": graph, "V": V, "ef": ef, "template": template, "tree_n": tree_n,
            "tree_seed": tree_seed, "n": n, "form": form, "mode": mode, "jobs": jobs}


def listed():
    return [
        # one coloring of a small template on a small graph: an interactive query, latency and launches
        _case("p3_s16", "rmat", 1 << 16, 16, "p3", 1),
        # the smallest graphs: a query on a neighbourhood of a few ten thousand vertices, ragged size
        _case("tree5_small", "rmat", 12345, 8, "tree5", 1),
        # the reference program's own flow (CountMat), a 5-tree over ten iterations on a million vertices
        _case("tree5_s20", "rmat", 1 << 20, 6, "tree5", 10, form="countmat"),
        # the same work in the batched form (colorings interleaved)
        _case("tree5_s20_groups", "rmat", 1 << 20, 6, "tree5", 10, form="groups"),
        # a 7-vertex template on the largest benchmark graph
        _case("spider7_s21", "rmat", 1 << 21, 8, "spider7", 2),
        # the headline template at a medium and at the headline size
        _case("tree12_s18", "rmat", 1 << 18, 8, "tree12", 1),
        _case("tree12_s20", "rmat", 1 << 20, 8, "tree12", 2),
        # double-precision tables: the high-precision mode of the headline template
        _case("tree12_s17_fp64", "rmat", 1 << 17, 8, "tree12", 1, mode="fp64"),
        # a graph without hubs (all degrees near the mean), odd size, a random 9-vertex tree
        _case("tree9_uniform", "uniform", 200003, 10, "random", 1, tree_n=9, tree_seed=11),
        # the reference's operation order for every product, odd size, a random 8-vertex tree
        _case("tree8_exact", "rmat", 100003, 12, "random", 2, mode="exact", tree_n=8, tree_seed=3),
        # a stream of different templates of 3 to 10 vertices on one graph, one coloring each
        _case("jobs_s16", "rmat", 1 << 16, 8, "mixed", 1, form="jobs", tree_seed=5, jobs=32),
        # a new graph every pass: host CSC arrays to the GPU, one coloring, the graph dropped
        _case("upload_tree5_s18", "rmat", 1 << 18, 8, "tree5", 1, form="upload"),
    ]


def _flops(case):
    return work(case)["flops"]


def draw(rng):
    most = max(_flops(c) for c in listed())
    while True:
        graph = rng.choice(["rmat", "rmat", "rmat", "uniform"])
        V = int(2 ** rng.uniform(13, 21))
        ef = rng.randint(4, 16)
        form = rng.choice(["plain", "plain", "plain", "groups", "jobs", "upload", "countmat"])
        mode = rng.choice(["fp32", "fp32", "fp32", "exact", "fp64"])
        if form in ("countmat", "upload"):
            mode = "fp32"
        template = rng.choice(["p3", "tree5", "spider7", "tree12", "random", "random", "random"])
        c = _case("", graph, V, ef, template, rng.randint(1, 6), form, mode, rng.randint(3, 9), rng.randrange(1 << 16))
        if form == "jobs":
            c.update(template="mixed", n=1, jobs=rng.randint(4, 40))
        if template != "random" or form == "jobs":
            c["tree_n"] = 0
        if form == "upload":
            c["n"] = 1
        # doubles cost twice the bytes; graphs of many colors stay below the largest listed case
        if _flops(c) * (2 if mode == "fp64" else 1) <= most:
            del c["name"]
            return c


# ---------------------------------------------------------------------------
# templates

def _random_tree(n, rng):
    """A uniform random labelled tree (Pruefer sequence, smallest leaf first)."""
    seq = [rng.randrange(n) for _ in range(n - 2)]
    deg = [1] * n
    for a in seq:
        deg[a] += 1
    edges = []
    for a in seq:
        leaf = min(i for i in range(n) if deg[i] == 1)
        edges.append((leaf, a))
        deg[leaf] -= 1
        deg[a] -= 1
    u, v = [i for i in range(n) if deg[i] == 1]
    return n, edges + [(u, v)]


def _templates(case):
    """The (k, edges) of a pass: one template, or one per job."""
    rng = random.Random(case["tree_seed"])
    if case["form"] == "jobs":
        return [_random_tree(rng.randint(3, 10), rng) for _ in range(case["jobs"])]
    if case["template"] == "random":
        return [_random_tree(case["tree_n"], rng)]
    return [TEMPLATES[case["template"]]]


def _steps(n, edges):
    """The template's DP rooted at vertex 0: (vertex, child, size before, size of
    the child's subtree) in the order in which the subtrees are joined."""
    adj = [[] for _ in range(n)]
    for a, b in edges:
        adj[a].append(b)
        adj[b].append(a)
    out = []

    def down(x, parent):
        size = 1
        for y in adj[x]:
            if y != parent:
                s = down(y, x)
                out.append((x, y, size, s))
                size += s
        return size

    down(0, -1)
    return out


# ---------------------------------------------------------------------------
# graphs

_edges = {}   # the data sets of this process (edges on the GPU), the last few


def _dataset(case):
    """The undirected edges (u < v, each once) of the case's graph, on the GPU."""
    key = (case["graph"], case["V"], case["ef"])
    if key not in _edges:
        V, m = case["V"], case["V"] * case["ef"]
        gen = torch.Generator(device="cuda").manual_seed(1)
        if case["graph"] == "uniform":
            u = torch.randint(0, V, (m,), generator=gen, device="cuda")
            v = torch.randint(0, V, (m,), generator=gen, device="cuda")
        else:
            # R-MAT (0.57, 0.19, 0.19, 0.05) over the next power of two, names
            # scrambled; the names at or past V are folded back
            scale = max(1, (V - 1).bit_length())
            u = torch.zeros(m, dtype=torch.int64, device="cuda")
            v = torch.zeros(m, dtype=torch.int64, device="cuda")
            for _ in range(scale):
                r = torch.rand(m, generator=gen, device="cuda")
                u = u * 2 + (r >= 0.76)
                v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
            name = torch.randperm(1 << scale, generator=gen, device="cuda")
            u, v = name[u] % V, name[v] % V
        keep = u != v
        k = torch.unique(torch.minimum(u, v)[keep] * V + torch.maximum(u, v)[keep])
        while len(_edges) > 3:
            _edges.pop(next(iter(_edges)))
        _edges[key] = (k // V, k % V)
    return _edges[key]


def _renamed(case, seed):
    """The data set's edges with the vertices renamed by the seed, on the GPU."""
    u, v = _dataset(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    name = torch.randperm(case["V"], generator=gen, device="cuda")
    return name[u], name[v]


def _seed_base(seed):
    return (int(seed) * 7919 + 13) & 0x7FFFFFFF


# ---------------------------------------------------------------------------
# the cases' contract

def prepare(case, seed):
    u, v = _renamed(case, seed)
    src, dst = u.to(torch.int32).cpu().numpy(), v.to(torch.int32).cpu().numpy()
    V, form = case["V"], case["form"]
    s = {"case": case, "seed": _seed_base(seed), "templates": [sg.Graph(*t) for t in _templates(case)]}
    if form == "countmat":
        csc = sg.CSCGraph()
        csc.createFromEdgeListFile(V, len(src), src, dst)
        s["csc"] = csc
        s["cm"] = sg.CountMat()
        s["cm"].initialization(None, csc, 1, case["n"])
        s["cm"].set_seed(s["seed"])
        return s
    g = sg.DeviceGraph.from_edges(V, src, dst)
    if form == "upload":
        s["offsets"], s["neighbors"] = g.csc()
    else:
        s["graph"] = g
    return s


def run(s):
    c, form, t = s["case"], s["case"]["form"], s["templates"]
    mode = sg.MODE_FP64 if c["mode"] == "fp64" else sg.MODE_REFERENCE
    exact = c["mode"] == "exact"
    if form == "countmat":
        estimate = s["cm"].compute(t[0])
        return {"estimate": estimate, "raw": s["cm"].raw_counts()}
    if form == "jobs":
        return {"raw": sg.count_jobs(s["graph"], t, [s["seed"] + j for j in range(len(t))], mode=mode, exact=exact)}
    g = sg.DeviceGraph(s["offsets"], s["neighbors"]) if form == "upload" else s["graph"]
    return {"raw": sg.count(g, t[0], c["n"], s["seed"], mode=mode, exact=exact, batch=c["n"] if form == "groups" else 0)}


def work(case):
    """Per coloring and join of a subtree of m vertices to one of p: the
    adjacency is read once, every table's entries that can be non-zero (the
    color sets holding the vertex's own color) once, the result written once;
    an add for each neighbour and such entry without the vertex's color, a
    multiply-add for each pair of sets that split the result's set."""
    V, nnz, es = case["V"], 2 * case["ef"] * case["V"], 8 if case["mode"] == "fp64" else 4
    nbytes, flops = 0, 0
    for k, edges in _templates(case):
        for _, _, p, m in _steps(k, edges):
            rows = [math.comb(k - 1, x - 1) if x > 1 else 1 for x in (p, m, p + m)]
            nbytes += 4 * (V + 1 + nnz) + es * V * (sum(rows) if p + m < k else rows[0] + rows[1] + 1)
            flops += nnz * (math.comb(k - 2, m - 1) if m > 1 else 1)
            flops += 2 * V * math.comb(k - 1, p + m - 1) * math.comb(p + m - 1, p - 1)
    return {"bytes": nbytes * case["n"], "flops": flops * case["n"]}


def _colors(V, k, seed):
    """rand() % k after srand(seed), one draw per vertex: the C library's own."""
    libc = ctypes.CDLL(None)
    rand = libc.rand
    libc.srand(ctypes.c_uint(seed & 0xFFFFFFFF))
    return torch.tensor([rand() % k for _ in range(V)], dtype=torch.int64, device="cuda")


def _colorful(adj, V, n, edges, colors):
    """The number of color-preserving embeddings with all colors different, in
    64 bits: tables [color sets][V] of every rooted subtree."""
    sets = {m: [s for s in range(1 << n) if bin(s).count("1") == m] for m in range(1, n + 1)}
    at = {m: {s: i for i, s in enumerate(sets[m])} for m in sets}
    one = torch.zeros(n, V, dtype=torch.float64, device="cuda")
    one.scatter_(0, colors[None, :], 1.0)
    table = {x: one for x in range(n)}
    for x, y, p, m in _steps(n, edges):
        child = table.pop(y)
        agg = torch.sparse.mm(adj, child.t().contiguous()).t().contiguous()
        del child
        main, out = table[x], torch.zeros(len(sets[p + m]), V, dtype=torch.float64, device="cuda")
        for i, s in enumerate(sets[p + m]):
            sub = s
            while sub:   # the subsets of s
                if sub in at[m]:
                    out[i].addcmul_(main[at[p][s ^ sub]], agg[at[m][sub]])
                sub = (sub - 1) & s
        table[x] = out
    return float(table[0].sum())


def exact(case, seed):
    u, v = _renamed(case, seed)
    V = case["V"]
    row, col = torch.cat([u, v]), torch.cat([v, u])
    order = torch.argsort(row * V + col)
    off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(row, minlength=V), 0)
    adj = torch.sparse_csr_tensor(off, col[order], torch.ones(len(row), dtype=torch.float64, device="cuda"), (V, V))
    # the reference scales the first table by the float 1e-12 and the sum by 1e12
    scale = 1.0 if case["mode"] == "fp64" else float(np.float32(1e-12)) * 1e12
    base, ts = _seed_base(seed), _templates(case)
    if case["form"] == "jobs":
        todo = [(t, base + j) for j, t in enumerate(ts)]
    else:
        todo = [(ts[0], base + i) for i in range(case["n"])]
    raw = [_colorful(adj, V, k, edges, _colors(V, k, sd)) * scale for (k, edges), sd in todo]
    out = {"raw": np.array(raw, np.float64)}
    if case["form"] == "countmat":
        k = ts[0][0]
        out["estimate"] = math.floor(float(np.mean(raw)) / (math.factorial(k) / k ** k) + 0.5)
    return out
