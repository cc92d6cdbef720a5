"""Graphs unlike the R-MAT ones: a few very long lists, dense graphs, lists of
every length at which the work is split another way.  Counts against the
general path (raw counts agree to the FP64 sum's rounding, below 1e-12), and
times against it where the default form once was slower."""
import time

import numpy as np
import pytest

import subgraph_b200 as sg
from tests.helpers import TEMPLATES, rel
from tests.test_gpu_rooted import _both, _csc

pytestmark = pytest.mark.gpu


def _hubs(n, leaves):
    """n vertices joined to all of `leaves`, which are a ring."""
    e = [(h, n + i) for h in range(n) for i in range(leaves)]
    return _csc(n + leaves, e + [(n + i, n + (i + 1) % leaves) for i in range(leaves)])


def _clique(n):
    return _csc(n, [(i, j) for i in range(n) for j in range(i)])


def _degrees(degs):
    """A vertex of each degree; their neighbours have up to three, one of the next one's among them."""
    e, at = [], len(degs)
    for v, d in enumerate(degs):
        e += [(v, at + i) for i in range(d)]
        e += [(at + i, at + i + 1) for i in range(0, d - 1, 3)] + [(at - 1, at)] * (v > 0)
        at += d
    return _csc(at, e)


GRAPHS = {
    "few hubs": lambda: _hubs(3, 600),         # their items go one to an SM
    "many hubs": lambda: _hubs(160, 600),      # more items than SMs
    "clique": lambda: _clique(300),            # all vertices past the hub threshold: no hubs where rows are wide
    "degrees": lambda: _degrees([1, 2, 3, 7, 8, 9, 10, 15, 16, 17, 31, 32, 33, 63, 64, 255, 256, 257, 1023, 1024, 1025, 1026]),
}


@pytest.mark.parametrize("graph", GRAPHS)
def test_counts_equal_general_path(graph):
    g = GRAPHS[graph]().device_graph()
    trees = [(k, [(i, i + 1) for i in range(k - 1)]) for k in (2, 3, 4, 5, 6, 8, 9, 10, 12)]
    for k, edges in trees + [TEMPLATES["spider7"], TEMPLATES["tree12"]]:
        t = sg.Graph(k, edges)
        for kw in (dict(exact=True), dict(mode=sg.MODE_FP64)):
            a, b = _both(g, t, 2, 5 + k, autotune=False, **kw)
            assert (k > 5 or np.all(a > 0)) and all(rel(x, y) <= 1e-12 for x, y in zip(a, b)), (k, edges, kw, a, b)


@pytest.mark.parametrize("ring", [37880, 37888, 37889, 60001])
def test_many_vertices_of_few_neighbours(ring):
    """More of them than SMs x 256 (37,888 on 148) take two threads each; their lists
    have one to eight entries, beside longer ones."""
    rng = np.random.default_rng(ring)
    e = [(i, (i + 1) % ring) for i in range(ring)]
    e += [(int(v), (int(v) + j) % ring) for v in rng.integers(0, ring, ring // 8) for j in range(2, 2 + int(v) % 4)]
    e += [(ring, i) for i in range(0, 3000, 2)] + [(ring + 1, i) for i in range(20)] + [(0, ring + 2)]
    g = _csc(ring + 4, e).device_graph()
    for k, edges in [(k, [(i, i + 1) for i in range(k - 1)]) for k in (2, 3, 5, 9)] + [TEMPLATES["star4"], TEMPLATES["spider7"]]:
        t = sg.Graph(k, edges)
        for kw in (dict(exact=True), dict(mode=sg.MODE_FP64)):
            a, b = _both(g, t, 1, 3 + k, autotune=False, **kw)
            assert a[0] > 0 and rel(a[0], b[0]) <= 1e-12, (k, edges, kw, a, b)


def _edges(V, src, dst):
    return sg.DeviceGraph.from_edges(V, src.astype(np.int32), dst.astype(np.int32))


def _best(g, t, **kw):
    for _ in range(2):
        sg.count(g, t, 1, 5, **kw)
    ms = []
    for _ in range(8):
        t0 = time.perf_counter()
        sg.count(g, t, 1, 5, **kw)
        ms.append((time.perf_counter() - t0) * 1e3)
    return min(ms)


# ms of the two on one B200: 20 lists of 100,000, 7-spider 3.08 (1.53 with the items
# spread over the SMs) against 1.87; 2000 vertices all joined, path of 10 2.64 (1.48
# without hubs) against 1.95
@pytest.mark.parametrize("graph, template", [("lists", "spider7"), ("clique", "path10")])
def test_no_slower_than_general_path(graph, template):
    if graph == "lists":
        rng = np.random.default_rng(1)
        g = _edges(200000, rng.integers(0, 20, 2000000), rng.integers(0, 200000, 2000000))
    else:
        g = _edges(2000, *np.triu_indices(2000, 1))
    t = sg.Graph(*TEMPLATES[template]) if template in TEMPLATES else sg.Graph(10, [(i, i + 1) for i in range(9)])
    a, b = _best(g, t), _best(g, t, flat=False)
    assert a <= 1.1 * b, (a, b)
