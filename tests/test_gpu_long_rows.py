"""Rows around the length that one warp walks before the rest is dealt to the
grid in parts (128, 256, 512 or 2,048 arcs by the graph's size): hubs of every
length next to a first part and to the parts behind it, on the persistent
solver (its knobs select it), below and above the first two sizes; and
the allocation-free solve with as many rows past the first part as fit its
scratch.  Flows are integers that the input determines: no tolerance."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu

LENGTHS = [126, 127, 128, 129, 130, 255, 256, 257, 383, 384, 385, 511, 512, 513, 640, 641, 767, 769, 2048, 2049]


def _hubs(pad, seed):
    """s -> hub -> middle -> second -> t for every hub; `pad` arcs apart from it.
    The hubs get more, less or as much as their middles let through."""
    rng = np.random.default_rng(seed)
    tail, head, cap = [], [], []
    nxt, value, t = 2, 0, 1
    for i, k in enumerate(LENGTHS):
        hub, mid, sec = nxt, np.arange(k) + nxt + 1, np.arange(k) + nxt + 1 + k
        nxt += 1 + 2 * k
        open_ = rng.integers(0, 3, k)
        give = [int(open_.sum()), int(open_.sum()) + 7, max(1, int(open_.sum()) - 5)][i % 3]
        tail += [[0], np.full(k, hub), mid, sec]
        head += [[hub], mid, sec, np.full(k, t)]
        cap += [[give], np.full(k, 2), open_, np.full(k, 3)]
        value += min(give, int(open_.sum()))
    extra = max(2, pad // 8)
    tail.append(nxt + rng.integers(0, extra, pad))
    head.append(nxt + rng.integers(0, extra, pad))
    cap.append(np.ones(pad, int))
    return W.Graph.from_arcs(nxt + extra, np.concatenate(tail), np.concatenate(head), np.concatenate(cap), 0, t), value


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("pad", [0, 2_200_000, 8_600_000])
def test_hubs_of_every_length(pad, layout):
    g, value = _hubs(pad, 5 + pad)
    with W.DeviceGraph(g, layout) as d:
        for algo, tile in (("vc", 8), ("vc", 32), ("tc", 0)):
            # gr_rounds: a knob of the persistent solver for every pair
            assert d.solve(algo, tile=tile, gr_rounds=20).flow == value
            rep = d.verify()
            assert rep["ok"] and rep["cut_value"] == value


@pytest.mark.parametrize("degree", [129, 150])
def test_noalloc_with_the_most_long_rows(degree):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(degree)
    hubs = 510_000 // (degree + 1)
    i = np.repeat(np.arange(hubs), degree)
    j = (i + np.tile(np.arange(degree) * 7, hubs)) % hubs  # every row on both sides has `degree` arcs
    tail = np.concatenate([np.zeros(hubs, int), i + 2, np.arange(hubs) + 2 + hubs])
    head = np.concatenate([np.arange(hubs) + 2, j + 2 + hubs, np.ones(hubs, int)])
    cap = np.concatenate([rng.integers(1, 400, hubs), rng.integers(0, 4, hubs * degree), rng.integers(1, 400, hubs)])
    g = W.Graph.from_arcs(2 + 2 * hubs, tail, head, cap, 0, 1)
    assert g.n <= 65_536 and 2 * g.m <= 1 << 20
    off, dst, c, back = W.build_bcsr(g)
    arc = torch.from_numpy(np.stack([dst, c], 1)).cuda()
    arx = torch.from_numpy(np.stack([back, c], 1).astype(np.int32)).cuda()
    row = torch.from_numpy(off).cuda()
    flow = C.c_int64(-1)
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    for algo in (0, 1):
        assert W.lib().wbpr_solve_bcsr_noalloc(g.n, 2 * g.m, row.data_ptr(), arc.data_ptr(), arx.data_ptr(), g.s, g.t, algo,
                                               None, C.byref(flow)) == 0
        assert flow.value == want
