"""Steps that only save time, on a device without the memory for them: the copy
of the arcs in play (lump64.cu), the work list of deep refinements
(deep_kernels.cuh), the one-launch refinement itself (fused.cu) of a graph that has
the buffers of the other path.  The call goes on without them."""
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


def _short_of(spare, call):
    """call's result on an empty device, and on one that lacks `spare` of the
    bytes which that took (a context keeps its blocks)."""
    import torch
    with R.Context(0) as ctx:
        call(ctx)  # (the kernels are loaded)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with R.Context(0) as ctx:
        want = call(ctx)
        used = free - torch.cuda.mem_get_info()[0]
    assert used > 2 * spare
    hog = torch.empty(torch.cuda.mem_get_info()[0] - used + spare, dtype=torch.uint8, device="cuda")
    try:
        with R.Context(0) as ctx:
            got = call(ctx)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert (got.blocks, got.rounds, got.verified) == (want.blocks, want.rounds, 1) and np.array_equal(got.labels, want.labels)
    return got, want


def test_no_room_for_the_arcs_in_play():
    off, idx, wt = _half_twins(1 << 17, 64)  # the copy takes 16 bytes for half of 8 M arcs
    got, want = _short_of(4 * len(idx), lambda ctx: ctx.refine_f64(off, idx, wt))
    assert got.kernel_launches != want.kernel_launches


def test_no_room_for_the_work_list():
    n, k = 1 << 20, 300  # the list takes some 76 bytes per node, most of them after the launch's own
    off = np.minimum(np.arange(n + 1), k).astype(np.uint64)
    idx = np.arange(1, k + 1, dtype=np.uint32)
    got, want = _short_of(30 << 20, lambda ctx: ctx.refine(off, idx))
    assert want.rounds == k + 1 and got.kernel_launches < want.kernel_launches


def test_no_room_for_the_one_launch_refinement():
    import torch
    off, idx = G.er_directed(1 << 20, 1 << 21, seed=3)
    with R.Context(0) as ctx:
        one = ctx.refine(off, idx)
        ctx.trim()
        ctx.set_opts(persistent=False)
        g = ctx.upload(off, idx)
        want = g.refine()
        ctx.set_opts(persistent=True)
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = g.refine()
        finally:
            del hog
            torch.cuda.empty_cache()
        again = g.refine()
        g.free()
    assert got.kernel_launches > again.kernel_launches == one.kernel_launches
    for r in (one, got, again):
        assert (r.blocks, r.rounds, r.verified) == (want.blocks, want.rounds, 1) and np.array_equal(r.labels, want.labels)
