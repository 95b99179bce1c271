"""Phase 2 and the cut searches on the persistent kernel: on one block (graphs of
up to 16,384 units; a row of over 4,096 arcs keeps their searches from the
shared-memory solvers), and on a grid of blocks for power-law graphs too large for
a cluster.  Both extreme minimum cuts and the completed flow are the oracle's."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _bundle(n, arcs, seed):
    """A random graph, one vertex of which has `arcs` arcs, most of them parallel."""
    rng = np.random.default_rng(seed)
    m = 6 * n
    hub, k = n // 2, arcs // 2
    return W.Graph.from_arcs(n, np.r_[rng.integers(0, n, m), np.full(k, hub), rng.integers(0, n, k)],
                             np.r_[rng.integers(0, n, m), rng.integers(0, n, k), np.full(k, hub)],
                             rng.integers(0, 30, m + 2 * k), 0, n - 1)


CASES = {
    "one block, few vertices": lambda: _bundle(12, 5000, 1),
    "one block": lambda: _bundle(60, 6000, 2),
    "one block, sparse": lambda: _bundle(500, 4300, 3),
    "a grid of blocks": lambda: W.gen_rmat(14, 40, seed=5),
    "a grid, longer rows": lambda: W.gen_rmat(16, 16, seed=6),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
def test_cuts_and_the_completed_flow(name, layout):
    g = CASES[name]()
    flow, sink_ind, source_ind = oracle.mincut(g.n, g.off, g.dst, g.cap, g.s, g.t)
    tail = np.repeat(np.arange(g.n), np.diff(g.off))
    inner = np.ones(g.n, bool)
    inner[[g.s, g.t]] = False
    with W.DeviceGraph(g, layout) as d:
        for algo in ("vc", "tc"):
            assert d.solve(algo).flow == flow and d.verify()["ok"]
            assert np.array_equal(d.mincut_adjoint(0)[0], sink_ind)
            to_sink = d.cut_sides(0)
            assert np.array_equal((to_sink[tail] == 0) & (to_sink[g.dst] == 1), sink_ind != 0)
            assert np.array_equal(d.mincut_adjoint(1)[0], source_ind)  # completes the flow first
            _, e, f = d.read_state()
            assert ((f >= 0) & (f <= g.cap)).all() and not e[inner].any()
            net = np.zeros(g.n, np.int64)
            np.add.at(net, g.dst, f)
            np.add.at(net, tail, -f.astype(np.int64))
            assert not net[inner].any() and net[g.t] == flow
