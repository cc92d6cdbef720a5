"""Offsets that fall are refused wherever they do (before any device is asked for:
this file runs without a GPU)."""
import numpy as np
import pytest

import subgraph_b200 as sg


@pytest.mark.parametrize("V", [2, 3, 4, 5, 8, 9, 33, 1000])
def test_falling_offsets_are_refused(V):
    good = np.arange(V + 1, dtype=np.int32) * 2
    nbr = np.zeros(2 * V, np.int32)
    for v in {1, V // 2, V - 1} - {0}:
        off = good.copy()
        off[v] = off[v + 1] + 1
        with pytest.raises(sg.SGError, match="offsets are not monotone"):
            sg.DeviceGraph(off, nbr)
    off = good.copy()
    off[1] = -1
    with pytest.raises(sg.SGError, match="offsets are not monotone"):
        sg.DeviceGraph(off, nbr)
