"""Sparse random graphs on both sides of the size at which single solves leave
the hybrid solver: the exact flow, the certificate and the sink side of the
cut, fresh, again on the restored residuals, and after new capacities."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("extra", [0, 1])
def test_both_sides_of_the_limit(extra, layout):
    n = 280_000
    m = ((1 << 22) - n) // 2 + extra  # n + 2 m = 2^22, the largest the hybrid solver takes, and one arc more
    rng = np.random.default_rng(extra)
    tail, head = rng.integers(0, n, m), rng.integers(0, n, m)
    tail[:200], head[200:400] = 0, n - 1
    g = W.Graph.from_arcs(n, tail, head, rng.integers(1, 30, m), 0, n - 1)
    assert g.m == m
    with W.DeviceGraph(g, layout) as d:
        for caps in (g.cap, rng.integers(0, 9, m).astype(np.int32)):
            d.set_capacities(caps)
            want, sink_side, _ = oracle.mincut(g.n, g.off, g.dst, caps, g.s, g.t)
            tails = np.repeat(np.arange(g.n), np.diff(g.off))
            for algo in ("vc", "tc"):
                assert d.solve(algo).flow == want
                rep = d.verify()
                assert rep["ok"] and rep["cut_value"] == want
                t_side = d.cut_sides(0).astype(bool)
                assert np.array_equal((~t_side[tails] & t_side[g.dst]).astype(np.int8), sink_side)
