"""Graphs whose flow goes through one long row: the shared-memory solvers walk it
with a warp or 8 lanes, the persistent kernel with the whole grid.  Such graphs
take no longer by default than on the persistent kernel (2 to 30 times as long
when size alone chose), in a handle, in a batch and in the caller's buffers;
long rows of the terminals, which no round walks, keep no graph from them.  The
bounds compare two times measured here and are wide: half as much again."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _rays(d, seed=6):
    """s -> hub -> d rays -> t: the hub's row has d + 1 arcs."""
    rng = np.random.default_rng(seed)
    mid = np.arange(d) + 2
    return W.Graph.from_arcs(d + 3, np.r_[0, np.full(d, 1), mid], np.r_[1, mid, np.full(d, d + 2)],
                             np.r_[3 * d, rng.integers(0, 6, d), rng.integers(0, 6, d)], 0, d + 2)


def _median(f, k=9):
    return float(np.median([f() for _ in range(k)][2:]))


def _seconds(f):
    t = time.perf_counter()
    f()
    return time.perf_counter() - t


# 20,000: the cluster's shared memory would hold it; 29,000 and 60,000: the hybrid solver's size
@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("rays", [9000, 20000, 29000, 60000])
def test_a_hub_goes_to_the_persistent_kernel(rays, layout):
    g = _rays(rays)
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    with W.DeviceGraph(g, layout) as d:
        assert d.solve("vc").flow == d.solve("vc", resident=-1).flow == want and d.verify()["ok"]
        assert _median(lambda: d.solve("vc").solve_ms) < 1.5 * _median(lambda: d.solve("vc", resident=-1).solve_ms)
        best, _ = d.autotune("vc")
        assert best.resident == 0
        # another terminal pair: the hub itself is one, and its row is no obstacle
        assert d.solve("vc", 1, g.t).flow == oracle.dinic(g.n, g.off, g.dst, g.cap, 1, g.t) and d.verify()["ok"]


def test_a_batch_of_hubs_goes_to_the_general_kernel():
    graphs = [_rays(10000, k) for k in range(8)]
    want = [oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t) for g in graphs]
    with W.Batch(graphs) as b:
        assert b.solve()[0].tolist() == want
        ours = _median(lambda: b.solve()[1])
        assert b.solve(batch_cluster=-1)[0].tolist() == want
        assert ours < 1.3 * _median(lambda: b.solve(batch_cluster=-1)[1])


@pytest.mark.parametrize("rays", [12000, 20000])
def test_a_hub_in_the_callers_buffers(rays):
    torch = pytest.importorskip("torch")
    g = _rays(rays)
    off, dst, cap, back = W.build_bcsr(g)
    row = torch.from_numpy(off).cuda()
    arc = torch.from_numpy(np.stack([dst, cap], 1)).cuda()
    arx = torch.from_numpy(np.stack([back, cap], 1).astype(np.int32)).cuda()
    flow = C.c_int64(-1)

    def solve():
        assert W.lib().wbpr_solve_bcsr_noalloc(g.n, 2 * g.m, row.data_ptr(), arc.data_ptr(), arx.data_ptr(), g.s, g.t, 1,
                                               None, C.byref(flow)) == 0

    solve()
    assert flow.value == oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    with W.DeviceGraph(g, "bcsr") as d:
        persistent = _median(lambda: _seconds(lambda: d.solve("vc", resident=-1)), 15)
    assert _median(lambda: _seconds(solve), 15) < 1.5 * persistent


def test_long_rows_of_the_terminals_do_not_matter():
    g = W.gen_grid(150, 160, 2)  # 24,000 arcs at each terminal
    want = oracle.fifo_pr(g.n, g.off, g.dst, g.cap, g.s, g.t)
    with W.DeviceGraph(g, "bcsr") as d:
        assert d.solve("vc").flow == want and d.verify()["ok"]
        assert 1.5 * _median(lambda: d.solve("vc").solve_ms, 5) < _median(lambda: d.solve("vc", resident=-1).solve_ms, 5)
