"""Calls that ask for device memory beyond what their handle holds, when there
is none: what another path can do without it is done there.  The checked build
refuses pool requests from a given size on; nothing is really exhausted.  Run in
a process of its own, which loads that build."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = r"""
import ctypes as C, sys
sys.path[:0] = [%r, %r]
import numpy as np
import oracle
import wbpr_gb300 as W

def refuse(from_bytes):
    f = W.lib().wbpr_checked_refuse_from
    f.argtypes, f.restype = [C.c_int64], None
    f(from_bytes)

def exact(g):
    return oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t)
""" % (ROOT, os.path.join(ROOT, "tests"))


def run(body):
    r = subprocess.run([sys.executable, "-c", HEAD + body], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, WBPR_CHECKED="1"))
    assert r.returncode == 0, r.stdout[-1000:] + r.stderr[-3000:]


def test_a_solve_without_room_for_arc_records():
    run(r"""
for layout in ("bcsr", "rcsr"):
    g = W.gen_layered(31, 641, 3, 6, 1, 1000, 8)  # the hybrid solver's: 16 bytes a residual arc
    with W.DeviceGraph(g, layout) as d:
        refuse(1 << 20)
        assert d.solve("vc").flow == exact(g) and d.verify()["ok"]
        held = d.device_bytes
        refuse(0)
        assert d.solve("vc").flow == exact(g) and d.verify()["ok"] and d.device_bytes == held
""")


def test_cut_sides_without_any_room():
    run(r"""
for make in (lambda: W.gen_genrmf(6, 6, 1, 500, 2), lambda: W.gen_rmat(15, 8, seed=3)):
    g = make()
    _, sink, source = oracle.mincut(g.n, g.off, g.dst, g.cap, g.s, g.t)
    tail = np.repeat(np.arange(g.n), np.diff(g.off))
    for layout in ("bcsr", "rcsr"):
        with W.DeviceGraph(g, layout) as d:
            d.solve("vc")
            refuse(1)
            to_sink, from_source = d.cut_sides(0), d.cut_sides(1)
            assert np.array_equal((to_sink[tail] == 0) & (to_sink[g.dst] == 1), sink != 0)
            assert np.array_equal((from_source[tail] == 1) & (from_source[g.dst] == 0), source != 0)
            refuse(0)
            assert d.solve("vc").flow == exact(g) and d.verify()["ok"]
""")


def test_a_batch_without_room_for_arc_records():
    run(r"""
graphs = [W.gen_layered(31, 641, 3, 6, 1, 1000, 8), W.gen_grid(90, 80, 1), W.gen_genrmf(24, 20, 1, 10000, 5),
          W.gen_genrmf(6, 9, 1, 10000, 2)]
want = [exact(g) for g in graphs]
with W.Batch(graphs) as b:
    held = b.device_bytes
    refuse(1)
    assert b.solve()[0].tolist() == want and b.device_bytes == held
    refuse(0)
    assert b.solve(max_ms=60000.0)[0].tolist() == want and b.device_bytes > held  # another capture, with room
""")


def test_a_batch_holds_one_set_of_records():
    """A split that asks for more records than the last one leaves only its own
    behind.  (Four clusters of 16 blocks, or of one, hold four times the largest
    instance's arcs; two and two hold less.)"""
    run(r"""
graphs = [W.gen_grid(100 + 10 * k, 90, k) for k in range(4)]
want = [exact(g) for g in graphs]
splits = (graphs[2].n + 2 * graphs[2].m, 1)  # from so many units on an instance has the largest cluster
alone = []
for c in splits:
    with W.Batch(graphs) as one:
        assert one.solve(batch_cluster=c)[0].tolist() == want
        alone.append(one.device_bytes)
assert alone[0] < alone[1]
for order in (splits, splits[::-1]):
    with W.Batch(graphs) as b:
        for c in order:
            assert b.solve(batch_cluster=c)[0].tolist() == want
        assert b.device_bytes == alone[1], (b.device_bytes, alone)
""")
