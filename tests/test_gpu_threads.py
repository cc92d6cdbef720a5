"""Different graph handles used from different threads: every kernel is launched
with the shared-memory size its template and graph ask for, from several
threads at once, and each count is the one a single thread gets."""
import random
import threading

import pytest

import subgraph_b200 as sg
from tests.test_gpu_rooted import _csc, _wheel

pytestmark = pytest.mark.gpu


def _ring(n, reach):
    """Every vertex of degree 2 * reach: no hubs."""
    return _csc(n, [(i, (i + j) % n) for i in range(n) for j in range(1, reach + 1)])


# the default form, and the general path (its tuning would only take time here)
@pytest.mark.parametrize("general, calls", [(False, 1500), (True, 200)])
def test_counts_from_several_threads_equal_serial(general, calls):
    form = dict(flat=False, autotune=False) if general else {}
    # with hubs and without: the same kernels at different sizes
    graphs = [_wheel(1700, 400, 1).device_graph(), _ring(400, 4).device_graph(), _wheel(900, 100, 2).device_graph(),
              _ring(300, 3).device_graph()]
    trees = [(k, [(i, i + 1) for i in range(k - 1)]) for k in (4, 5, 6, 7, 8, 9, 10)]
    kinds = [{}, dict(mode=sg.MODE_FP64), dict(exact=True)]
    templates = [[sg.Graph(*t) for t in trees] for _ in graphs]
    want = [[[sg.count(g, t, 1, 7, **kw, **form)[0] for t in ts] for kw in kinds] for g, ts in zip(graphs, templates)]
    wrong = []

    def work(i):
        rng = random.Random(i)
        for _ in range(calls):
            q, j = rng.randrange(len(kinds)), rng.randrange(len(trees))
            try:
                got = sg.count(graphs[i], templates[i][j], 1, 7, **kinds[q], **form)[0]
            except sg.SGError as e:
                got = str(e)
            if got != want[i][q][j]:
                wrong.append((i, q, j, got, want[i][q][j]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(graphs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:5])
