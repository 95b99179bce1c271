"""The resident solver (the residual graph in the shared memory of one block
or of a 16-block cluster) and the hybrid one (its vertices there, its arcs in
global memory) at the sizes where their split can go wrong, against
the oracle and against the persistent kernel (which any of its own knobs, such
as `tile`, selects): exact flow, valid labels and the device certificate, both
extreme minimum cuts, and the completed flow, on both layouts and algorithms.
Every compared value is an integer that the input determines: no tolerance."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _random(n, m, top, seed):
    rng = np.random.default_rng(seed)
    return W.Graph.from_arcs(n, rng.integers(0, n, m), rng.integers(0, n, m), rng.integers(0, top, m), 0, n - 1)


def _star(rays, seed):
    """s -> hub -> rays -> t: one row of 2 * rays arcs and no other long one."""
    rng = np.random.default_rng(seed)
    mid = np.arange(rays) + 2
    tail = np.concatenate([[0], np.full(rays, 1), mid])
    head = np.concatenate([[1], mid, np.full(rays, rays + 2)])
    cap = np.concatenate([[3 * rays], rng.integers(0, 6, rays), rng.integers(0, 6, rays)])
    return W.Graph.from_arcs(rays + 3, tail, head, cap, 0, rays + 2)


CASES = {
    "two vertices": lambda: W.Graph.from_arcs(2, [0, 0, 1], [1, 1, 0], [3, 4, 5], 0, 1),
    "no arcs": lambda: W.Graph.from_arcs(33, [], [], [], 0, 32),
    "isolated vertices": lambda: W.Graph.from_arcs(4000, [0, 7, 3999], [7, 3999, 0], [9, 5, 2], 0, 3999),
    "a group less one": lambda: _random(31, 120, 9, 1),
    "a group and one": lambda: _random(33, 150, 9, 2),
    "a block's warps and one": lambda: _random(1025, 6000, 50, 3),
    "the largest single block": lambda: W.gen_genrmf(10, 26, 1, 10000, 1),
    "the smallest cluster": lambda: W.gen_genrmf(10, 29, 1, 10000, 2),
    "largest capacities": lambda: W.Graph.from_arcs(3, [0, 1], [1, 2], [2**31 - 1, 2**31 - 1], 0, 2),
    "a long row in one block": lambda: _star(700, 4),
    "long rows in a cluster": lambda: W.gen_rmat(13, 14, seed=5),
    "a row of several blocks' arcs": lambda: _star(29000, 6),  # fits no block: the persistent kernel takes it
    "a cluster nearly full": lambda: W.gen_layered(64, 480, 3, 6, 1, 1000, 7),
    "hybrid": lambda: W.gen_layered(31, 641, 3, 6, 1, 1000, 8),
    "hybrid, every vertex active at once": lambda: W.gen_layered(3, 30011, 3, 6, 1, 1000, 9),
    "hybrid, rows in global memory": lambda: W.gen_grid(431, 419, 10),
    "the largest hybrid": lambda: W.gen_layered(20, 14233, 3, 6, 1, 50, 11),  # 284,662 vertices of at most 284,672
    "one more than the largest hybrid": lambda: W.gen_layered(5, 56935, 3, 6, 1, 50, 12),
    "a deep path over a cluster": lambda: W.Graph.from_arcs(9000, np.arange(8999), np.arange(1, 9000),
                                                            np.full(8999, 3), 0, 8999),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
def test_resident_solver_agrees(name, layout):
    g = CASES[name]()
    flow, sink_ind, source_ind = oracle.mincut(g.n, g.off, g.dst, g.cap, g.s, g.t)
    tail = np.repeat(np.arange(g.n), np.diff(g.off))
    inner = np.ones(g.n, bool)
    inner[[g.s, g.t]] = False
    with W.DeviceGraph(g, layout) as d:
        # resident, persistent, resident again: each starts from what the other left
        for algo, tune in (("vc", {}), ("vc", dict(tile=8)), ("tc", {})):
            r = d.solve(algo, **tune)
            assert r.flow == flow, (algo, tune)
            rep = d.verify()
            assert rep["ok"] and rep["label_violations"] == 0, (algo, tune, rep)
            h, e, f = d.read_state()
            assert h.min() >= 0 and h.max() <= g.n and e[g.t] == flow
            stranded = int(((e > 0) & (h >= g.n) & inner).sum())
            assert r.stranded == stranded
            assert np.array_equal(d.mincut_adjoint(0)[0], sink_ind)
            assert np.array_equal(d.mincut_adjoint(1)[0], source_ind)  # completes the flow first
            _, e, f = d.read_state()
            assert ((f >= 0) & (f <= g.cap)).all() and not e[inner].any()
            net = np.zeros(g.n, np.int64)
            np.add.at(net, g.dst, f)
            np.add.at(net, tail, -f.astype(np.int64))
            assert not net[inner].any() and net[g.t] == flow


def test_resident_budgets_and_new_terminals():
    g = W.gen_genrmf(12, 16, 1, 10000, 3)
    with W.DeviceGraph(g, "bcsr") as d:
        for kw in (dict(max_rounds=2), dict(max_ms=1e-6)):
            with pytest.raises(W.WbprError) as e:
                d.solve("vc", **kw)
            assert e.value.status == 3
            assert d.solve("vc").flow == oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
        assert d.solve("vc", 5, g.n - 7).flow == oracle.dinic(g.n, g.off, g.dst, g.cap, 5, g.n - 7)
        cap = np.random.default_rng(1).integers(0, 500, g.m).astype(np.int32)
        d.set_capacities(cap)
        assert d.solve("vc", g.s, g.t).flow == oracle.dinic(g.n, g.off, g.dst, cap, g.s, g.t)


@pytest.mark.parametrize("make", [lambda: W.gen_genrmf(6, 9, 1, 10000, 2), lambda: W.gen_rmat(13, 16, seed=8),
                                  lambda: W.gen_grid(80, 90, 3), lambda: W.gen_rmat(14, 16, seed=9)])
def test_caller_buffers_on_either_solver(make):
    """wbpr_solve_bcsr_noalloc on graphs of one block, of a cluster and too
    large for one, twice, and with the same buffers refused in between."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    g = make()
    off, dst, cap, back = W.build_bcsr(g)
    arc = torch.from_numpy(np.stack([dst, cap], 1)).cuda()
    row = torch.from_numpy(off).cuda()
    flow = C.c_int64(-1)

    def solve(twins, algo):
        arx = torch.from_numpy(np.stack([twins, cap], 1).astype(np.int32)).cuda()
        return W.lib().wbpr_solve_bcsr_noalloc(g.n, 2 * g.m, row.data_ptr(), arc.data_ptr(), arx.data_ptr(), g.s, g.t, algo,
                                               None, C.byref(flow))

    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    unpaired = back.copy()
    unpaired[3] = 2 * g.m
    for algo in (0, 1):
        assert solve(back, algo) == 0 and flow.value == want
        assert solve(unpaired, algo) == 1 and b"twin" in W.lib().wbpr_last_error()
