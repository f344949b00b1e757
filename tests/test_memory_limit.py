"""Double weights when the device has no room for the copy of the arcs in play
(lump64.cu), which only saves time: the call goes on without it."""
import numpy as np
import pytest

import rbsc_b200 as R
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


def _half_twins(n, d):
    """Rows of d arcs; the second quarter repeats the first (its nodes stay in
    play), the other half ends up alone (its arcs are dropped)."""
    rng = np.random.default_rng(7)
    heads = rng.integers(0, n, size=(n, d))
    wt = rng.random(size=(n, d))
    q = n // 4
    heads[q: 2 * q], wt[q: 2 * q] = heads[:q], wt[:q]
    off = np.arange(n + 1, dtype=np.uint64) * np.uint64(d)
    return off, heads.astype(np.uint32).ravel(), wt.ravel()


def test_no_room_for_the_arcs_in_play():
    import torch
    off, idx, wt = _half_twins(1 << 17, 64)  # the copy takes 16 bytes for half of 8 M arcs
    with R.Context(0) as ctx:
        ctx.refine_f64(off, idx, wt)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with R.Context(0) as ctx:
        want = ctx.refine_f64(off, idx, wt)
        used = free - torch.cuda.mem_get_info()[0]  # the context keeps its blocks
    copy = 16 * len(idx) // 2
    assert used > 2 * copy
    hog = torch.empty(torch.cuda.mem_get_info()[0] - used + copy // 2, dtype=torch.uint8, device="cuda")
    try:
        with R.Context(0) as ctx:
            r = ctx.refine_f64(off, idx, wt)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert (r.blocks, r.rounds, r.verified) == (want.blocks, want.rounds, 1) and np.array_equal(r.labels, want.labels)
    assert r.kernel_launches != want.kernel_launches  # (the copies' launches)
