"""The undo log when its slots fill.  A warp writes to one of 256 slots of 4,096
entries (on graphs of up to 2^21 arcs), so a solve on one or two blocks has 8 or 16
of them and fills these within a few rounds; the next fresh solve must then rewrite
every residual.  Every solve is exact and certified, whatever came before."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 2])
def test_solves_after_a_full_log(blocks):
    g = W.gen_grid(90, 90, 5)
    other = W.Graph(g.n, g.off, g.dst, np.roll(g.cap, 17), g.s, g.t)
    want, turned = (oracle.dinic(x.n, x.off, x.dst, x.cap, x.s, x.t) for x in (g, other))
    with W.DeviceGraph(g, "bcsr") as d:
        for k in range(3):
            r = d.solve("vc", grid_blocks=blocks)
            assert r.pushes > blocks * 8 * 4096  # more than these slots hold: one at least is full
            assert r.flow == want
            rep = d.verify()
            assert rep["ok"] and rep["label_violations"] == 0
            if k == 1:  # a solve on the whole grid, whose log does not fill, in between
                assert d.solve("vc", grid_blocks=76, resident=-1).flow == want and d.verify()["ok"]
        d.complete_flow()
        assert d.solve("vc", grid_blocks=blocks).flow == want and d.verify()["ok"]
        d.set_capacities(other.cap)
        for _ in range(2):
            assert d.solve("vc", grid_blocks=blocks).flow == turned and d.verify()["ok"]
