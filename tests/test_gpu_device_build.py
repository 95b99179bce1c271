"""The device build on graphs that are small but for their vertices: more than
20,000 of them send a graph of any number of arcs through it, so its refusals and
the corner cases of its sort and length classes are reached with a few arcs.
Entry for entry against the host builder."""
import numpy as np
import pytest

import wbpr_gb300 as W
from conftest import graph_of
from test_gpu_builder import random_graph, same_as_host

pytestmark = pytest.mark.gpu

N = 20001


def padded(g, where):
    """The graph with N isolated vertices before, behind, or between its own."""
    at = {"before": N + np.arange(g.n), "behind": np.arange(g.n), "between": (np.arange(g.n) * (N // g.n + 1))}[where]
    tail = at[np.repeat(np.arange(g.n), np.diff(g.off))]
    return W.Graph.from_arcs(max(N, int(at.max()) + 1) + N, tail, at[g.dst], g.cap, int(at[g.s]), int(at[g.t]))


@pytest.mark.parametrize("where", ["before", "behind", "between"])
def test_golden_cases_among_isolated_vertices(golden, where):
    for case in golden:
        if case["n"] >= 2 and case["s"] != case["t"]:
            same_as_host(padded(graph_of(case), where))


@pytest.mark.parametrize("n,m", [(N, 0), (N, 1), (N, 40), (N, 4095), (N, 4096), (N, 4097), (65536, 300), (65537, 300), (30, 20001)])
def test_random_shapes(n, m):
    same_as_host(random_graph(n, m, n + m))


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
def test_incoming_capacities_past_int32(layout):
    k, top = 100, 2**31 - 1
    rng = np.random.default_rng(1)
    # one head whose 100 arcs span several warps of the sorted order, others around it
    tail, head = np.r_[np.zeros(k, int), np.full(40, 2), rng.integers(0, N, 300)], np.r_[np.full(k, 1), np.full(40, 3), rng.integers(4, N, 300)]
    cap = np.r_[np.full(k, top // k), np.full(340, 7)]
    cap[0] += top - int(cap[:k].sum())
    order = rng.permutation(tail.size)

    def graph(c):
        return W.Graph.from_arcs(N, tail[order], head[order], c[order], 0, 3)

    same_as_host(graph(cap))  # at the limit exactly
    for at in (0, k - 1):
        over = cap.copy()
        over[at] += 1
        with pytest.raises(W.WbprError) as e:
            W.DeviceGraph(graph(over), layout)
        assert e.value.status == 4


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("fault", ["capacity first", "capacity last", "offsets decrease", "offsets start", "head"])
def test_invalid_input_is_refused(fault, layout):
    g = random_graph(N, 5000, 3)
    off, dst, cap = g.off.copy(), g.dst.copy(), g.cap.copy()
    if fault == "capacity first":
        cap[0] = -1
    elif fault == "capacity last":
        cap[-1] = -2**31
    elif fault == "offsets decrease":
        v = int(np.flatnonzero(np.diff(off))[7])
        off[v + 1] = off[v] - 1
    elif fault == "offsets start":
        off[0] = 1
    else:
        dst[2500] = N
    with pytest.raises(W.WbprError) as e:
        W.DeviceGraph(W.Graph(N, off, dst, cap, 0, N - 1), layout)
    assert e.value.status == 1
    same_as_host(g)
