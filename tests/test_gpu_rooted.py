"""Rooted rows (the default plain form) against the general path: a call with
one of the general path's forms switched off takes the full-width tables, and
in exact mode (and in FP64) both sum the same products in the same order, so
raw counts agree to the FP64 sum's rounding (at most 2^20 terms with Kahan
compensation: below 1e-12)."""
import random

import numpy as np
import pytest

import subgraph_b200 as sg
from oracle import oracle as O
from tests.helpers import TEMPLATES, prufer_tree, rel

pytestmark = pytest.mark.gpu


def _csc(V, edges):
    src = np.array([e[0] for e in edges], np.int32)
    dst = np.array([e[1] for e in edges], np.int32)
    csc = sg.CSCGraph()
    csc.createFromEdgeListFile(V, len(edges), src, dst)
    return csc


def _wheel(n, extra, seed):
    """Vertex 0 joined to all others, the others a cycle, some chords, then a
    pendant path and an isolated vertex: one long list, degrees 1 to 5."""
    rng = random.Random(seed)
    e = [(0, i) for i in range(1, n)] + [(i, i + 1) for i in range(1, n - 1)] + [(1, n - 1)]
    e += [(rng.randrange(1, n), rng.randrange(1, n)) for _ in range(extra)]   # self loops and duplicates among them
    e += [(n - 1, n), (n, n + 1)]
    return _csc(n + 3, e)


def _both(g, t, n, seed, **kw):
    return sg.count(g, t, n, seed, **kw), sg.count(g, t, n, seed, flat=False, rooted=False, hub_threshold=0, **kw)


# every width of aggregate and row: one lane to several column blocks a vertex
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13])
def test_rooted_rows_equal_general_path(k):
    rng = random.Random(100 + k)
    trees = [[(i, i + 1) for i in range(k - 1)]]   # the general path's FP64 tiles hold no more than a path's at 13
    if k < 13:
        trees += [prufer_tree(k, rng) for _ in range(3)]
    el = sg.rmat(9, 8, seed=k)
    rm = sg.CSCGraph()
    rm.createFromEdgeListFile(el.getNumVertices(), el.getNumEdges(), el.getSrcList(), el.getDstList())
    for csc in (rm, _wheel(1700, 400, k)):
        g = csc.device_graph()
        for edges in trees:
            t = sg.Graph(k, edges)
            for kw in (dict(exact=True), dict(mode=sg.MODE_FP64)):
                a, b = _both(g, t, 2, 3 + k, **kw)
                assert all(rel(x, y) <= 1e-12 for x, y in zip(a, b)), (k, edges, kw, a, b)


@pytest.mark.parametrize("n", [2, 3, 4, 31, 32, 33, 257])
def test_rooted_rows_small_graphs(n):
    """Tiles, chunks and lists at their smallest, against the oracle."""
    csc = _wheel(n, n // 2, n)
    g = csc.device_graph()
    for k, edges in (TEMPLATES["p3"], TEMPLATES["tree5"], (4, [(0, 1), (0, 2), (0, 3)]), (6, [(i, i + 1) for i in range(5)])):
        P = O.Plan(k, edges)
        raw = sg.count(g, sg.Graph(k, edges), 3, 11, exact=True)
        for i in range(3):
            want = O.count_coloring(csc.getIndexCol(), csc.getIndexRow(), P, O.colors(11 + i, csc.getNumVertices(), k))
            assert (raw[i] == want == 0) or rel(raw[i], want) <= 1e-12, (n, k, i, raw[i], want)


def test_rooted_rows_asymmetric_adjacency():
    """Lists that are not symmetric: the rows of vertices of degree 1 are read by
    others than their own neighbour and may not be left out."""
    rng = np.random.default_rng(5)
    V = 300
    deg = rng.integers(0, 4, V)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    nbr = rng.integers(0, V, off[-1]).astype(np.int32)
    g = sg.DeviceGraph(off, nbr)
    for k, edges in (TEMPLATES["tree5"], TEMPLATES["spider7"], (3, [(0, 1), (1, 2)])):
        a, b = _both(g, sg.Graph(k, edges), 4, 9, exact=True)
        assert np.any(a > 0)
        assert all(x == y or rel(x, y) <= 1e-12 for x, y in zip(a, b)), (k, a, b)


@pytest.mark.parametrize("n", [1, 2, 5, 9])
def test_colorings_in_flight_equal_one_by_one(n):
    csc = _wheel(1700, 400, 2)
    g = csc.device_graph()
    t = sg.Graph(*TEMPLATES["spider7"])
    many = sg.count(g, t, n, 40)
    for i in range(n):
        assert many[i] == sg.count(g, t, 1, 40 + i)[0]
    assert np.array_equal(many, sg.count(g, t, n, 40, batch=n))
