"""Graphs that fit a cluster's shared memory by size but not as they split, with
rows of 8,000 arcs where the blocks' shares end: the kernel finds out, changes
nothing, and the persistent kernel solves, on a handle and in the caller's
buffers, as often as it is asked."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _lumps(seed):
    """410,000 residual arcs over 16 blocks: 25,600 each, of at most 27,200, in rows of 8,000."""
    rng = np.random.default_rng(seed)
    n, lumps = 2000, 40
    hub = np.arange(20, n, n // lumps)[:lumps]
    tail = np.repeat(hub, 3900)
    head = hub[rng.integers(0, lumps, tail.size)]  # among themselves: 3,900 out and about as many in
    m = 205000 - tail.size
    return W.Graph.from_arcs(n, np.r_[tail, rng.integers(0, n, m)], np.r_[head, rng.integers(0, n, m)],
                             rng.integers(0, 50, 205000), 0, n - 1)


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
def test_a_split_that_does_not_fit(layout):
    g = _lumps(1)
    row = np.diff(g.off) + np.bincount(g.dst, minlength=g.n)
    # as the kernel splits: a block's share begins at the first vertex with its part of the weight before it
    before = np.r_[0, np.cumsum(14 + 8 * row)]
    first = [int(np.searchsorted(before[:-1], before[-1] * k // 16)) for k in range(17)]
    arcs = np.r_[0, np.cumsum(row)]
    assert row.max() <= 8192 and max(8 * (arcs[first[k + 1]] - arcs[first[k]]) for k in range(16)) > 227 * 1024 - 14336
    rule = W.lib()._ZN8wbpr_dev16resident_clusterExx
    rule.argtypes, rule.restype = [C.c_longlong, C.c_longlong], C.c_int
    assert rule(g.n, 2 * g.m) == 16
    flow, sink_ind, source_ind = oracle.mincut(g.n, g.off, g.dst, g.cap, g.s, g.t)
    with W.DeviceGraph(g, layout) as d:
        for _ in range(2):
            assert d.solve("vc").flow == flow and d.verify()["ok"]
            assert np.array_equal(d.mincut_adjoint(0)[0], sink_ind)
            assert np.array_equal(d.mincut_adjoint(1)[0], source_ind)


def test_in_the_callers_buffers():
    torch = pytest.importorskip("torch")
    g = _lumps(2)
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    off, dst, cap, back = W.build_bcsr(g)
    row = torch.from_numpy(off).cuda()
    arc = torch.from_numpy(np.stack([dst, cap], 1)).cuda()
    arx = torch.from_numpy(np.stack([back, cap], 1).astype(np.int32)).cuda()
    flow = C.c_int64(-1)
    for algo in (0, 1, 1):
        assert W.lib().wbpr_solve_bcsr_noalloc(g.n, 2 * g.m, row.data_ptr(), arc.data_ptr(), arx.data_ptr(), g.s, g.t, algo,
                                               None, C.byref(flow)) == 0
        assert flow.value == want
