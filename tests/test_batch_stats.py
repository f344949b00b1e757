"""The copies of a batch's results are in its statistics, on both ways to them
(one block per graph; a sort when a graph is too large for that)."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large", [False, True], ids=["block per graph", "sort"])
def test_time_of_the_copies(large):
    parts = [G.er_directed(n, 4 * n, seed=n) for n in ([700] * 200 + ([2049] if large else []))]
    gn = np.concatenate([[0], np.cumsum([len(o) - 1 for o, _ in parts])]).astype(np.uint64)
    off = np.concatenate([[0]] + [np.diff(o.astype(np.int64)) for o, _ in parts]).cumsum().astype(np.uint64)
    idx = np.concatenate([i + np.uint32(b) for (_, i), b in zip(parts, gn)]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        for r in (ctx.batch_refine(off, idx, gn), g.batch_refine(gn)):
            assert np.array_equal(r.colors, ex.labels)
            assert r.stats.d2h_bytes == 4 * len(ex.labels) and 0 < r.stats.d2h_ms < 1e3 * r.stats.time_s
        g.free()
