"""Graphs with few long rows on the persistent kernel, where a row of up to 2,048
arcs is walked by one warp to its end, and with as many or as long rows as make
it cut them into parts: exact and certified on either side of both limits, on both
layouts and in the caller's buffers."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _hubs(count, arcs, seed):
    """A sparse random graph, `count` of whose vertices have `arcs` arcs at least."""
    rng = np.random.default_rng(seed)
    n, m = 20000, 60000
    hub = rng.choice(np.arange(1, n - 1), count, replace=False)
    out = np.repeat(hub, arcs // 2)
    back = np.repeat(hub, arcs - arcs // 2)
    tail = np.r_[rng.integers(0, n, m), out, rng.integers(0, n, back.size), np.zeros(40, int), rng.integers(0, n, 40)]
    head = np.r_[rng.integers(0, n, m), rng.integers(0, n, out.size), back, rng.choice(hub, 40), np.full(40, n - 1)]
    return W.Graph.from_arcs(n, tail, head, rng.integers(1, 60, tail.size), 0, n - 1)


@pytest.mark.parametrize("count,arcs", [(1, 120), (1, 129), (1, 500), (1, 2030), (1, 2060), (4, 1000), (30, 300), (34, 300), (1, 9000)])
def test_exact_on_either_side_of_the_limits(count, arcs):
    g = _hubs(count, arcs, count + arcs)
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    for layout in ("bcsr", "rcsr"):
        with W.DeviceGraph(g, layout) as d:
            for algo in ("vc", "tc"):
                assert d.solve(algo, resident=-1).flow == want
                rep = d.verify()
                assert rep["ok"] and rep["label_violations"] == 0
    torch = pytest.importorskip("torch")
    off, dst, cap, back = W.build_bcsr(g)
    row = torch.from_numpy(off).cuda()
    arc = torch.from_numpy(np.stack([dst, cap], 1)).cuda()
    arx = torch.from_numpy(np.stack([back, cap], 1).astype(np.int32)).cuda()
    flow = C.c_int64(-1)
    for _ in range(2):
        assert W.lib().wbpr_solve_bcsr_noalloc(g.n, 2 * g.m, row.data_ptr(), arc.data_ptr(), arx.data_ptr(), g.s, g.t, 1, None,
                                               C.byref(flow)) == 0
        assert flow.value == want
