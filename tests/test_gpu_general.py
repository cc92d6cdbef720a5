"""The general path (full-width tables), which a call takes with one of its forms
switched off and the table helpers with a hub threshold, against the
reference's tables and against the default form: tables and root values bit
for bit, raw counts to the FP64 sum's rounding (at most 2^20 terms with Kahan
compensation: below 1e-12)."""
import ctypes
import random

import numpy as np
import pytest

import subgraph_b200 as sg
from oracle import oracle as O
from subgraph_b200._lib import CountOpts, check
from tests.helpers import TEMPLATES, prufer_tree, rel
from tests.test_gpu_parity import dev_graph, sha

pytestmark = pytest.mark.gpu
NO_HUBS = 1 << 30   # the general path without hub rows
FORMS = [dict(flat=False), dict(rooted=False), dict(blocked=False), dict(flat=False, rooted=False, blocked=False)]


def _trees(seed, n):
    rng = random.Random(seed)
    return [TEMPLATES["tree12"], TEMPLATES["spider7"], TEMPLATES["tree5"]] + \
           [(k, prufer_tree(k, rng)) for k in [rng.randint(4, 12) for _ in range(n)]]


@pytest.mark.parametrize("hub_threshold", [8, NO_HUBS])
def test_tables_bit_exact(golden, hub_threshold):
    n = 0
    for c in golden.cases:
        if not c.table_sha:
            continue
        g, _, _ = dev_graph(golden, c.graph)
        t = sg.Graph(c.n, c.edges)
        for s, digest in c.table_sha.items():
            assert sha(sg.debug_sub_table(g, t, c.seed, s, hub_threshold=hub_threshold)) == digest, (c.key, s)
            n += 1
        assert sg.debug_root(g, t, c.seed, hub_threshold=hub_threshold)[1] == c.raw[0], c.key
    assert n > 30


@pytest.mark.parametrize("mode", [sg.MODE_REFERENCE, sg.MODE_FP64])
def test_tables_and_roots_equal_default_form(golden, mode):
    for gname in ("rmat10", "rmat12"):
        g, _, _ = dev_graph(golden, gname)
        for k, edges in _trees(11, 4):
            t = sg.Graph(k, edges)
            want, raw = sg.debug_root(g, t, 6, mode=mode)
            for thr in (16, NO_HUBS):
                got, raw2 = sg.debug_root(g, t, 6, mode=mode, hub_threshold=thr)
                assert np.array_equal(got, want) and raw == raw2, (gname, k, edges, thr)
            subs = sum(1 for _ in t.shared_tables())
            for s in range(1, subs):
                a = sg.debug_sub_table(g, t, 6, s, mode=mode)
                assert np.array_equal(a, sg.debug_sub_table(g, t, 6, s, mode=mode, hub_threshold=16)), (gname, k, edges, s)


@pytest.mark.parametrize("mode", [sg.MODE_REFERENCE, sg.MODE_FP64])
@pytest.mark.parametrize("batch", [0, 4])
def test_counts_of_each_form(golden, mode, batch):
    """Plain and in interleaved groups, with hub rows and without, tuned for one of them."""
    g, _, _ = dev_graph(golden, "rmat12")
    for i, (k, edges) in enumerate(_trees(13, 2)):
        t = sg.Graph(k, edges)
        want = sg.count(g, t, 5, 21, mode=mode, exact=True)
        for form in FORMS:
            for thr in (0, 32):
                got = sg.count(g, t, 5, 21, mode=mode, exact=True, batch=batch, hub_threshold=thr,
                               autotune=i == 2 and thr == 32, **form)
                assert all(rel(a, b) <= 1e-12 for a, b in zip(got, want)), (k, edges, form, thr, got, want)


@pytest.mark.parametrize("mode", [sg.MODE_REFERENCE, sg.MODE_FP64])
def test_job_streams(golden, mode):
    """Jobs with a form switched off (an option of the C interface), with hub rows
    and without, on fewer streams than jobs."""
    g, _, _ = dev_graph(golden, "rmat12")
    ts = [sg.Graph(*t) for t in _trees(17, 6)]
    seeds = np.arange(60, 60 + len(ts), dtype=np.uint32)
    want = sg.count_jobs(g, ts, seeds, mode=mode, exact=True)
    plans = (ctypes.c_void_p * len(ts))(*[t.plan for t in ts])
    for field in ("no_flat", "no_rooted", "no_blocked"):
        for thr, streams in ((0, 3), (32, 8)):
            o = CountOpts()
            sg.lib().sg_count_opts_default(ctypes.byref(o))
            o.mode, o.hub_threshold, o.exact, o.batch, o.no_autotune = mode, thr, 1, streams, 1
            setattr(o, field, 1)
            got = np.zeros(len(ts), np.float64)
            check(sg.lib().sg_count_jobs(g.handle, len(ts), ctypes.cast(plans, ctypes.c_void_p),
                                         seeds.ctypes.data_as(ctypes.c_void_p), ctypes.byref(o),
                                         got.ctypes.data_as(ctypes.c_void_p), None, None))
            assert all(rel(a, b) <= 1e-12 for a, b in zip(got, want)), (field, thr, got, want)


def test_overflowing_counts_are_infinite_in_every_form():
    """FP32 entries past the largest finite value (a vertex listing 259 others
    20,000 times each under a star of ten): no form skips or meets them differently."""
    V = 260
    adj = [np.tile(np.arange(1, V), 20000)] + [np.array([j for j in range(V) if j != i]) for i in range(1, V)]
    off = np.concatenate([[0], np.cumsum([len(a) for a in adj])]).astype(np.int32)
    g = sg.DeviceGraph(off, np.concatenate(adj).astype(np.int32))
    for edges in ([(0, 1), (0, 2)] + [(2, i) for i in range(3, 12)], [(0, i) for i in range(1, 12)],
                  [(0, 1), (1, 2), (1, 3)] + [(3, i) for i in range(4, 12)]):
        t = sg.Graph(12, edges)
        assert np.isfinite(sg.count(g, t, 1, 3, mode=sg.MODE_FP64)[0])
        for form in [{}, dict(batch=1)] + FORMS:
            raw = sg.count(g, t, 1, 3, exact=True, autotune=False, **form)[0]
            assert raw == np.inf, (edges, form, raw)


def test_template_that_only_the_general_path_takes(golden):
    """15 vertices, a path of 14 with a leaf at its eighth: a step of 6 and 2
    vertices whose rooted rows (3003 + 14 + 3432 columns, eight vertices a tile) do
    not fit shared memory where the general path's (5005 + 105 and a part of the
    outputs) do.  Plain, tuned and in groups, and jobs beside one that the default
    form would take."""
    g, col, row = dev_graph(golden, "rmat10")
    edges = [(i, i + 1) for i in range(13)] + [(7, 14)]
    t = sg.Graph(15, edges)
    P = O.Plan(15, edges)
    want = [O.count_coloring(col, row, P, O.colors(9 + i, len(col) - 1, 15)) for i in range(2)]
    raw, st = sg.count(g, t, 2, 9, exact=True, autotune=False, return_stats=True)
    assert all(rel(a, b) <= 1e-12 for a, b in zip(raw, want)), (raw, want)
    off, st2 = sg.count(g, t, 2, 9, exact=True, autotune=False, flat=False, return_stats=True)
    assert st["table_bytes"] == st2["table_bytes"] and np.array_equal(raw, off)
    for kw in (dict(autotune=True), dict(batch=2), dict(hub_threshold=16, autotune=False)):
        got = sg.count(g, t, 2, 9, exact=True, **kw)
        assert all(rel(a, b) <= 1e-12 for a, b in zip(got, want)), (kw, got, want)
    t5 = sg.Graph(*TEMPLATES["tree5"])
    got = sg.count_jobs(g, [t, t5, t], [9, 4, 10], exact=True)
    for a, b in zip(got, [want[0], sg.count(g, t5, 1, 4, exact=True)[0], want[1]]):
        assert rel(a, b) <= 1e-12, (got, want)
