"""Negative heads in graphs large enough for the device build: refused, and
the sort that runs before the refusal writes nothing outside its arrays."""
import numpy as np
import pytest

import wbpr_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["bcsr", "rcsr"])
@pytest.mark.parametrize("n", [200, 1000, 100_000])
@pytest.mark.parametrize("bad", ["first", "last", "tile", "every"])
def test_negative_heads_are_refused(n, bad, layout):
    rng = np.random.default_rng(n)
    m = 5 * 4096 + 4001
    off = np.sort(np.r_[0, rng.integers(0, m + 1, n - 1), m]).astype(np.int32)
    dst = rng.integers(0, n, m).astype(np.int32)
    cap = np.ones(m, np.int32)
    at = {"first": slice(0, 1), "last": slice(m - 1, m), "tile": slice(4096, 8192), "every": slice(0, m, 3)}[bad]
    dst[at] = -1 - (np.arange(m)[at] % 70_000).astype(np.int32)
    with pytest.raises(W.WbprError):
        W.DeviceGraph(W.Graph(n, off, dst, cap, 0, n - 1), layout)
    # and a good graph builds and solves afterwards
    g = W.gen_rmat(12, 8, seed=3)
    with W.DeviceGraph(g, layout) as d:
        d.solve("vc")
        assert d.verify()["ok"]
