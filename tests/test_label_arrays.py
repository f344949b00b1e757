"""A call that runs out of rounds leaves the caller's label array alone, and one
that does not fills it, whichever kernels refine the graph."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


def _graph(kind):
    if kind == "rows":  # the passes after the first signatures in one launch
        rng = np.random.default_rng(3)
        n, m = 300000, (1 << 22) + 5
        off, idx, _ = G.csr_from_arcs(n, rng.integers(0, n // 2, m), rng.integers(0, n, m), sort=False)
        return off, idx, (np.arange(n) % 3).astype(np.uint32)
    if kind == "deep":
        off, idx = G.path(300)
        s, d = G.arcs_of(off, idx)
        off, idx, _ = G.csr_from_arcs(9000, s, d)
        return off, idx, None
    n = dict(block=500, cluster=3000, grid=30000, phases=3000)[kind]
    off, idx = G.er_directed(n, 4 * n, seed=8)
    return off, idx, None


@pytest.mark.parametrize("kind", ["block", "cluster", "grid", "deep", "rows", "phases"])
def test_labels_only_after_success(kind):
    import torch
    off, idx, init = _graph(kind)
    ex = oracle.refine_exact(off, idx, None, init)
    n = len(off) - 1
    with R.Context(0, persistent=kind != "phases") as ctx:
        g = ctx.upload(off, idx)
        d_init = None if init is None else torch.from_numpy(init.view(np.int32)).cuda()
        out = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        call = lambda: g.refine_device(0 if init is None else d_init.data_ptr(), out.data_ptr())
        for rounds in sorted({1, ex.rounds - 1}):
            ctx.set_opts(max_rounds=rounds)
            with pytest.raises(R.RbscError, match="no fixpoint"):
                call()
            torch.cuda.synchronize()
            assert (out == -7).all()
        for rounds in (ex.rounds, 0):
            ctx.set_opts(max_rounds=rounds)
            out.fill_(-7)
            torch.cuda.synchronize()
            r = call()
            assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), ex.labels)
        g.free()
