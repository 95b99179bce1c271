"""The closure test of the matching kernel: closed sets (c + 1 left vertices on
c right ones, as a chain) of sizes around the limit it follows them to, rows
around the length it walks, next to a random part that keeps rounds and
relabels going.  The size must equal the oracle's, with valid labels and the
device certificate; every compared value is an integer: no tolerance."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _network(sizes, copies, width, seed):
    rng = np.random.default_rng(seed)
    left, right, nl, nr = [], [], 0, 0
    for c in sizes:
        for _ in range(copies):
            # left i knows rights i - 1 and i of its chain; `width` of them
            # also repeat their arcs to make longer rows (parallel arcs)
            for i in range(c + 1):
                for j in {max(i - 1, 0), min(i, c - 1)}:
                    for _ in range(width if i == 0 else 1):
                        left.append(nl + i)
                        right.append(nr + j)
            nl += c + 1
            nr += c
    n = 4000
    deg = np.minimum(rng.zipf(2.0, n), 60)
    left = np.concatenate([np.array(left, np.int64), nl + np.repeat(np.arange(n), deg)])
    right = np.concatenate([np.array(right, np.int64), nr + rng.integers(0, n, int(deg.sum()))])
    return W.bipartite_network(nl + n, nr + n, left, right)


@pytest.mark.parametrize("sizes,copies,width", [((1, 2, 3), 300, 1), ((14, 15, 16, 17), 120, 1), ((40, 200), 20, 1),
                                                ((1, 5), 200, 32), ((1, 5), 200, 33), ((16,), 1, 1)])
@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
def test_closed_sets(sizes, copies, width, layout):
    g = _network(sizes, copies, width, 7)
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    with W.DeviceGraph(g, layout) as d:
        for kw in ({}, dict(gr_plateau=1), dict(gr_rounds=3), dict(grid_blocks=4)):
            r = d.solve("vc", **kw)
            assert r.matching == 1 and r.flow == want, kw
            rep = d.verify()
            assert rep["ok"] and rep["label_violations"] == 0, (kw, rep)
            h, e, f = d.read_state()
            assert h.min() >= 0 and h.max() <= g.n and int(e.sum()) == want
