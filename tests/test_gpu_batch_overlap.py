"""The launches of a batch run side by side: instances on clusters (of the
hybrid solver, or of the general kernel where one of its knobs is set) and
instances on a block of the general kernel take together little more than the
longer kind alone.  Each kind's time is measured here, so the bound holds on any
device: one kind after the other would take the sum."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


def _clusters():
    """423,000 units each: a cluster on either solver."""
    return [W.gen_genrmf(30, 44, 1, 10000, seed) for seed in range(3)]


def _blocks():
    """A GENRMF too large for one block's shared memory, with too many long rows
    (of arcs without capacity) for the hybrid solver."""
    g = W.gen_genrmf(18, 30, 1, 10000, 9)
    rng = np.random.default_rng(1)
    tail = np.r_[np.repeat(np.arange(g.n), np.diff(g.off)), np.repeat(np.arange(100, 180), 40)]
    return [W.Graph.from_arcs(g.n, tail, np.r_[g.dst, rng.integers(0, g.n, 3200)], np.r_[g.cap, np.zeros(3200, int)],
                              g.s, g.t)]


def _time(graphs, want, tuning):
    with W.Batch(graphs) as b:
        ms = []
        for _ in range(6):
            flows, t = b.solve(**tuning)
            assert flows.tolist() == want
            ms.append(t)
    return float(np.median(ms[1:]))


@pytest.mark.parametrize("tuning", [{}, dict(tile=32)])
def test_kinds_of_instances_overlap(tuning):
    a, b = _clusters(), _blocks()
    wa, wb = ([oracle.fifo_pr(g.n, g.off, g.dst, g.cap, g.s, g.t) for g in x] for x in (a, b))
    ta, tb, both = _time(a, wa, tuning), _time(b, wb, tuning), _time(a + b, wa + wb, tuning)
    # the shorter kind hides behind the longer one, but for half of it
    assert both < max(ta, tb) + 0.5 * min(ta, tb), (ta, tb, both)
