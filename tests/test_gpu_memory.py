"""Device memory of the default form: colorings and jobs in flight where memory
is short, and graphs made and dropped one after another."""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

import subgraph_b200 as sg
from tests.helpers import TEMPLATES

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_jobs_fit_where_an_earlier_count_holds_memory():
    """The tables of an earlier count are no room for other buffers: with little
    free memory the jobs run on fewer streams and count the same."""
    torch = pytest.importorskip("torch")
    trees = [sg.Graph(*TEMPLATES["tree5"]), sg.Graph(*TEMPLATES["spider7"])]
    jobs = [trees[j % 2] for j in range(32)]
    seeds = list(range(32))
    small = sg.DeviceGraph.from_rmat(14, 8, seed=3)
    sg.count_jobs(small, jobs, seeds, streams=16)       # loads the kernels
    sg.count(small, sg.Graph(*TEMPLATES["tree12"]), 4, 1)
    other = sg.DeviceGraph.from_rmat(20, 8, seed=3)
    want = sg.count_jobs(other, jobs, seeds, streams=16)
    del other
    g = sg.DeviceGraph.from_rmat(20, 8, seed=3)         # 64 MB of neighbours a stream
    sg.count(g, sg.Graph(*TEMPLATES["tree12"]), 4, 1)   # 9 GB of tables
    torch.empty(1, device="cuda")
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = sg.count_jobs(g, jobs, seeds, streams=16)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)


CYCLES = """
import time
import subgraph_b200 as sg
from tests.helpers import TEMPLATES
t = sg.Graph(*TEMPLATES["tree12"])
el = sg.rmat(20, 8, seed=1)
csc = sg.CSCGraph()
csc.createFromEdgeListFile(el.getNumVertices(), el.getNumEdges(), el.getSrcList(), el.getDstList())
off, nbr = csc.getIndexCol(), csc.getIndexRow()
kept = sg.DeviceGraph(off, nbr)
sg.count(kept, t, 4, 3)
for _ in range(20):
    g = sg.DeviceGraph(off, nbr)
    for _ in range(2):
        t0 = time.perf_counter()
        sg.count(g, t, 4, 5)
        print((time.perf_counter() - t0) * 1e3)
    del g
"""


def test_graphs_made_and_dropped_reuse_their_memory():
    """A new graph of the same size finds the dropped one's memory: its first count
    does not wait for memory to be remapped (0.8 ms of 38 each time, and up to
    0.8 s at times).  In a process of its own, whose pool holds nothing else."""
    r = subprocess.run([sys.executable, "-c", CYCLES], capture_output=True, text=True, cwd=ROOT, timeout=120)
    assert r.returncode == 0, r.stderr
    ms = [float(x) for x in r.stdout.split()][4:]   # the first cycles grow the pool
    first, warm = sorted(ms[0::2]), sorted(ms[1::2])
    assert first[len(first) // 2] <= warm[len(warm) // 2] + 0.6, (first, warm)


def test_first_call_on_a_new_graph_is_a_warm_one():
    """Colorings in flight need streams and room for their tables: both are at hand
    when a graph of the same size was dropped before (an 8-vertex path on 2^17
    vertices: creating streams and asking the driver took a quarter of the call)."""
    t = sg.Graph(8, [(i, i + 1) for i in range(7)])
    el = sg.rmat(17, 9, seed=2)
    csc = sg.CSCGraph()
    csc.createFromEdgeListFile(el.getNumVertices(), el.getNumEdges(), el.getSrcList(), el.getDstList())
    off, nbr = csc.getIndexCol(), csc.getIndexRow()
    first, warm = [], []
    for _ in range(25):
        g = sg.DeviceGraph(off, nbr)
        for ms in (first, warm, warm, warm):
            t0 = time.perf_counter()
            sg.count(g, t, 4, 5)
            ms.append(time.perf_counter() - t0)
        del g
    assert sorted(first)[12] <= sorted(warm)[37] + 1.5e-4, (sorted(first)[12], sorted(warm)[37])


def test_first_call_with_a_new_template():
    """A template made, counted and dropped per call: its tables' memory comes from
    the pool (P3, R-MAT scale 16: 0.5 ms and up to 4.5 above the second call's
    0.1 with the driver's own allocations, 0.06 on full-width tables)."""
    g = sg.DeviceGraph.from_rmat(16, 16, seed=2)
    first, warm = [], []
    for _ in range(41):
        t = sg.Graph(*TEMPLATES["p3"])
        for ms in (first, warm):
            t0 = time.perf_counter()
            sg.count(g, t, 1, 5)
            ms.append((time.perf_counter() - t0) * 1e3)
        del t
    assert sorted(first)[20] <= sorted(warm)[20] + 0.25, (sorted(first)[20], sorted(warm)[20])
