"""The vertex sides of the two extreme minimum cuts, gathered on the device,
at the edges of a block and of the grid-stride loop.  Parallel paths
of two arcs have both cuts known in closed form, so the comparison is exact."""
import numpy as np
import pytest

import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("n", [2, 3, 31, 255, 256, 257, 1025, 155_648, 155_649, 311_300])
def test_sides_of_parallel_paths(n, layout):
    # s -> v -> t for every inner vertex v: by v mod 3 the first arc, the second
    # arc or both bind, and vertex n - 1 is the sink
    s, t = 0, n - 1
    v = np.arange(1, n - 1)
    if n == 2:
        g = W.Graph.from_arcs(2, [0], [1], [3], s, t)
        value = 3
    else:
        c1 = np.where(v % 3 == 0, 1, 2)
        c2 = np.where(v % 3 == 1, 1, 2)
        g = W.Graph.from_arcs(n, np.r_[np.zeros(n - 2, int), v], np.r_[v, np.full(n - 2, t)], np.r_[c1, c2], s, t)
        value = int(np.minimum(c1, c2).sum())
    sink = np.zeros(n, np.int8)
    src = np.zeros(n, np.int8)
    sink[t] = src[s] = 1
    # sink side: residual arc v -> t left (first arc binds); source side: s -> v left (second binds)
    sink[v] = v % 3 == 0
    src[v] = v % 3 == 1
    with W.DeviceGraph(g, layout) as d:
        assert d.solve("vc").flow == value
        for _ in range(2):
            assert np.array_equal(d.cut_sides(0), sink)
            assert np.array_equal(d.cut_sides(1), src)
