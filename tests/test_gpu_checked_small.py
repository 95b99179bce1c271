"""The bounds-checked build on the graphs that the shared-memory solvers take:
their records, slots and blocks are checked where they are used (an index out
of range is counted and the solve fails with WBPR_ERR_VERIFY), for one block, a
cluster and the hybrid solver, in every mode -- solve, the two cuts, the
completed flow, a batch -- and in the caller's own buffers.  The same graphs go
through the persistent kernel at its own grid size, one block up to 16,384
units (any of its knobs selects it).  Exact against the oracle: no tolerance."""
import json
import os
import subprocess
import sys

import pytest

import oracle
import wbpr_gb300 as W
from conftest import ROOT
from wbpr_gb300 import build as wb

SCRIPT = r"""
import ctypes as C, json, sys
sys.path.insert(0, %r)
import numpy as np
import wbpr_gb300 as W
exec(sys.stdin.read())
out = []
for make in MAKE:
    g = make()
    row = []
    for layout in ("bcsr", "rcsr"):
        with W.DeviceGraph(g, layout) as d:
            for kw in ({}, dict(gr_rounds=48)):
                row.append(int(d.solve("vc", **kw).flow))
                for side in (0, 1):  # side 1 completes the flow first
                    cut = d.cut_sides(side)
                    assert cut[g.s] == side and cut[g.t] == 1 - side
                    ind, _ = d.mincut_adjoint(side)
                    row.append(int(g.cap[ind != 0].astype(np.int64).sum()))
    out.append(row)
flows, _ = W.Batch([make() for make in MAKE]).solve()
print(json.dumps([out, [int(f) for f in flows]]))
"""
MAKE = r"""
def uniform(n, m, seed):
    rng = np.random.default_rng(seed)
    return W.Graph.from_arcs(n, rng.integers(0, n, m), rng.integers(0, n, m), rng.integers(0, 9, m), 0, n - 1)
MAKE = [lambda: W.Graph.from_arcs(2, [0, 0, 1], [1, 1, 0], [3, 4, 5], 0, 1),
        lambda: uniform(60, 400, 9), lambda: uniform(1025, 6000, 3),
        lambda: W.gen_genrmf(6, 6, 1, 500, 2), lambda: W.gen_genrmf(10, 29, 1, 10000, 2),
        lambda: W.gen_rmat(9, 16, seed=5), lambda: W.gen_rmat(13, 14, seed=5),
        lambda: W.gen_layered(64, 480, 3, 6, 1, 1000, 7), lambda: W.gen_layered(31, 641, 3, 6, 1, 1000, 8),
        lambda: W.gen_grid(24, 24, 1), lambda: W.gen_grid(431, 419, 10)]
"""


def test_every_solver_kernel_is_in_the_checked_build():
    assert {"pr_bcsr.cu", "pr_rcsr.cu", "resident.cu", "hybrid.cu"} <= set(wb.CHECKED_SOURCES)


@pytest.mark.gpu
def test_checked_shared_memory_solvers_stay_in_bounds():
    env = dict(os.environ, WBPR_CHECKED="1")
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT], input=MAKE, capture_output=True, text=True, env=env,
                       timeout=1200)
    assert r.returncode == 0, r.stderr[-3000:]
    rows, flows = json.loads(r.stdout.strip().splitlines()[-1])
    scope = {"W": W, "np": __import__("numpy")}
    exec(MAKE, scope)
    want = []
    for make in scope["MAKE"]:
        g = make()
        want.append(oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t))
    assert rows == [[v] * 12 for v in want]
    assert flows == want


def _alone(body):
    """Runs a program on the checked build in a process of its own."""
    head = "import sys\nsys.path[:0] = [%r, %r]\nimport numpy as np\nimport oracle\nimport wbpr_gb300 as W\n"
    r = subprocess.run([sys.executable, "-c", head % (ROOT, os.path.join(ROOT, "tests")) + body], capture_output=True,
                       text=True, env=dict(os.environ, WBPR_CHECKED="1"), timeout=1200)
    assert r.returncode == 0, r.stdout[-1000:] + r.stderr[-3000:]


@pytest.mark.gpu
def test_the_blocks_of_a_cluster_decide_alike():
    """When to relabel globally and when to give up hangs on a clock, which the
    lanes of a warp read at different times in this build: the blocks must all
    get one lane's answer.  Many relabels, and budgets that run out at any point."""
    _alone(r"""
for g in (W.gen_genrmf(8, 16, 1, 10000, 4), W.gen_genrmf(12, 20, 1, 10000, 3), W.gen_layered(31, 641, 3, 6, 1, 1000, 8)):
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    for layout in ("bcsr", "rcsr"):
        with W.DeviceGraph(g, layout) as d:
            for kw in [dict(max_ms=x) for x in (1e-3, 0.05, 0.2, 0.5)] + [dict(max_rounds=x) for x in (1, 5, 12)]:
                try:
                    assert d.solve("vc", **kw).flow == want
                except W.WbprError as e:
                    assert e.status == 3, e
            r = d.solve("vc")
            assert r.flow == want and r.global_relabels > 1 and d.verify()["ok"]
""")


@pytest.mark.gpu
def test_a_tile_works_on_one_value_of_the_excess():
    """Vertices that many others push to while their own tile pushes on: with the
    lanes of a tile apart, every unit must still be counted once."""
    _alone(r"""
rng = np.random.default_rng(5)
n, hubs = 3000, 24
tail, head = rng.integers(0, n, 30000), rng.integers(0, n, 30000)
tail[::3], head[1::3] = rng.integers(1, hubs, 10000), rng.integers(1, hubs, 10000)
for g in (W.Graph.from_arcs(n, tail, head, rng.integers(1, 1000, 30000), 0, n - 1), W.gen_rmat(10, 16, seed=4),
          W.gen_rmat(13, 12, seed=4), W.gen_genrmf(9, 9, 1, 100, 2), W.gen_grid(150, 170, 3)):
    want = oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
    tails = np.repeat(np.arange(g.n), np.diff(g.off))
    for layout in ("bcsr", "rcsr"):
        with W.DeviceGraph(g, layout) as d:
            for _ in range(3):
                assert d.solve("vc").flow == want and d.verify()["ok"]
                _, e, f = d.read_state()
                net = np.zeros(g.n, np.int64)
                np.add.at(net, g.dst, f)
                np.add.at(net, tails, -f.astype(np.int64))
                net[g.s] = e[g.s]
                assert (net == e).all()
""")
