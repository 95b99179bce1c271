"""Round and time budgets of the batched shared-memory solvers, reached with no
knob of the general kernel set: an instance that runs out reports -1 and the next
one is claimed by the same launch; the batch then solves exactly again."""
import numpy as np
import pytest

import oracle
import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1, 1 << 30])  # clusters as the batch needs, the largest, one block each
@pytest.mark.parametrize("budget", [dict(max_rounds=1), dict(max_rounds=9), dict(max_ms=1e-6), dict(max_ms=0.05)])
def test_budgets_are_reported_and_the_batch_recovers(budget, split):
    one_block = [W.gen_genrmf(6, 8, 1, 10000, k) for k in range(200)]  # more than there are SMs
    sparse = [W.gen_genrmf(14, 12, 1, 10000, k) for k in range(4)] + [W.gen_grid(90, 70, 1)]
    no_rounds = [W.Graph.from_arcs(3, [0], [1], [5], 0, 2)]
    graphs = one_block + sparse + no_rounds
    want = [oracle.dinic(g.n, g.off, g.dst, g.cap, g.s, g.t) for g in graphs]
    with W.Batch(graphs) as b:
        flows = np.zeros(b.count, np.int64)
        tuning = W.default_tuning(batch_cluster=split, **budget)
        import ctypes as C

        st = W.lib().wbpr_batch_solve(b._h, C.byref(tuning), flows.ctypes.data_as(C.POINTER(C.c_int64)), None)
        assert st == 3
        out = flows < 0
        assert out[:len(one_block) + len(sparse)].any() and not out[-1]
        assert all(f == w for f, w in zip(flows, want) if f >= 0)
        if "max_rounds" in budget and budget["max_rounds"] == 1:
            assert out[:-1].all()
        for _ in range(2):
            assert b.solve(batch_cluster=split)[0].tolist() == want
        assert b.solve(batch_cluster=split, max_rounds=1 << 20, max_ms=60000.0)[0].tolist() == want
