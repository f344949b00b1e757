"""Rows with more colours than a block's table of the exact check holds, or more
arcs than it may count, whose node shares its class: the one-launch refinements
decide them in a launch of their own (check_kernels.cuh) and do not start again."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


def _same(r, ex):
    assert r.done == 1 and r.verified == 1
    assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
    assert np.array_equal(r.labels, ex.labels)


def _hubs(k, copies, hubs, filler=0, seed=1):
    """hubs times `copies` nodes with the same k heads, in any order; the heads
    keep apart by their initial colours.  filler: arcs of other nodes."""
    rng = np.random.default_rng(seed)
    h = copies * hubs
    heads = 3 * k // 2
    rows = [rng.choice(heads, size=k, replace=False) + h for _ in range(hubs)]
    src = np.repeat(np.arange(h), k)
    dst = np.concatenate([rng.permutation(rows[i // copies]) for i in range(h)])
    n = h + heads
    init = np.concatenate([np.zeros(h), np.arange(1, heads + 1)]).astype(np.uint32)
    if filler:
        m = filler // 20
        src = np.concatenate([src, n + np.sort(rng.integers(0, m, filler))])
        dst = np.concatenate([dst, n + rng.integers(0, m, filler)])
        init = np.concatenate([init, np.full(m, heads + 1)]).astype(np.uint32)
        n += m
    off, idx, _ = G.csr_from_arcs(n, src, dst, sort=False)
    return off, idx, init


def _marked(off, idx, init, h, heads):
    """The same kept apart by arcs: head i points at the nodes of a chain that
    the bits of i name."""
    s, d = G.arcs_of(off, idx)
    n, bits = len(off) - 1, 14
    i, b = np.divmod(np.arange(heads * bits), bits)
    on = (i + 1) >> b & 1 == 1
    chain = n + np.arange(bits - 1)
    return G.csr_from_arcs(n + bits, np.concatenate([s, h + i[on], chain]), np.concatenate([d, n + b[on], chain + 1]), sort=False)[:2]


def _few_launches(off, idx, wt, init, most=16):
    """Every call decides the rows without the launch-per-phase path."""
    ex = oracle.refine_exact(off, idx, wt, init)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx, wt)
        for r in (ctx.refine(off, idx, wt, init), g.refine(init), g.refine(init)):
            _same(r, ex)
            assert r.kernel_launches <= most
        g.free()
    return ex


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("k", [1025, 2047, 2048, 2049, 4097, 70000])
def test_number_of_colours(k, weighted):
    off, idx, init = _hubs(k, 2, 1)
    wt = (idx % 5).astype(np.uint64) << np.uint64(60) if weighted else None
    _few_launches(off, idx, wt, init)


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
def test_many_wide_rows(weighted):
    off, idx, init = _hubs(6000, 4, 45)
    wt = (idx % 7 + 1).astype(np.uint64) if weighted else None
    ex = _few_launches(off, idx, wt, init)
    assert len(np.unique(ex.labels[:180])) == 45


@pytest.mark.parametrize("uniform", [False, True], ids=["colours", "uniform"])
def test_large_graphs(uniform):
    """The passes after the first signatures in one launch; resident from one
    class, the whole refinement."""
    off, idx, init = _hubs(5000, 3, 20, filler=1 << 22)
    if uniform:
        off, idx = _marked(off, idx, init, 60, 7500)
        init = None
    ex = _few_launches(off, idx, None, init, most=40)
    assert len(np.unique(ex.labels[:60])) == 20


def test_colours_of_no_weight():
    """Rows that differ in heads whose weights add up to 0 are equal."""
    k = 3000
    src = np.repeat([0, 1], k)
    dst = np.concatenate([np.arange(k) + 2, np.arange(k) + 2 + k // 3])
    wt = np.concatenate([np.where(np.arange(k) < k // 3, 0, 9), np.where(np.arange(k) < k - k // 3, 9, 0)])
    n = 2 + k + k // 3
    off, idx, w = G.csr_from_arcs(n, src, dst, wt)
    init = np.concatenate([[0, 0], np.arange(1, n - 1)]).astype(np.uint32)
    ex = _few_launches(off, idx, w, init)
    assert ex.labels[1] == 0


@pytest.mark.parametrize("n_short", [4000])
def test_long_member_beside_short_rows(n_short):
    """Reading the member's row once per short row would cost more than the
    launch-per-phase check, which decides here."""
    k = 3000
    src = np.concatenate([np.zeros(k + 1, np.int64), np.arange(1, n_short + 1)])
    dst = np.concatenate([n_short + 1 + np.arange(k + 1), np.full(n_short, n_short + 1 + k)])
    n = n_short + k + 2
    off, idx, w = G.csr_from_arcs(n, src, dst, np.where(dst == n - 1, 5, 0))
    init = np.concatenate([np.zeros(n_short + 1), np.arange(1, k + 2)]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, w, init)
    assert (ex.labels[: n_short + 1] == 0).all()
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx, w)
        for r in (ctx.refine(off, idx, w, init), g.refine(init), g.refine(init)):
            _same(r, ex)
        g.free()


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("more", [0, 30], ids=["wide", "wide and short"])
def test_differences_are_found(weighted, more):
    """No signatures: only the exact check tells rows apart, a wide one by its
    last head, short ones by their only one."""
    k = 5000
    src = np.concatenate([np.repeat([0, 1, 2], k), 3 + np.arange(more)])
    heads = np.arange(k)
    last = np.where(heads == k - 1, k, heads)
    dst = 3 + more + np.concatenate([heads, heads[::-1], last, np.arange(more)])
    n = 3 + more + k + 1
    off, idx, w = G.csr_from_arcs(n, src, dst, np.ones(len(src), np.uint64) if weighted else None, sort=False)
    init = np.concatenate([np.zeros(3 + more), np.arange(1, k + 2)]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, w, init)
    with R.Context(0, test_hash_bits=-1) as ctx:
        g = ctx.upload(off, idx, w)
        for r in (ctx.refine(off, idx, w, init), g.refine(init), g.refine(init)):
            assert r.verified == 1 and r.blocks == ex.blocks and np.array_equal(r.labels, ex.labels)
        g.free()


def _long_hubs(d, hubs, heads=300):
    """`hubs` nodes with d arcs each to the same few heads."""
    dst = hubs + np.arange(d, dtype=np.int64) * 7 % heads
    src = np.repeat(np.arange(hubs), d)
    off, idx, _ = G.csr_from_arcs(hubs + heads, src, np.tile(dst, hubs), sort=False)
    return off, idx, np.concatenate([np.zeros(hubs), 1 + np.arange(heads) % 40]).astype(np.uint32)


@pytest.mark.parametrize("kind", ["unit", "weighted", "uniform"])
@pytest.mark.parametrize("d", [540_000, 3_000_000])
def test_rows_of_more_arcs_than_a_block_counts(d, kind):
    """Shared by all warps: the first launch and three of the check's own (a
    call whose only work they are would otherwise wait for one block)."""
    off, idx, init = _long_hubs(d, 2, heads=1 if kind == "uniform" else 300)
    wt = (idx % 3 + 1).astype(np.uint64) if kind == "weighted" else None
    init = None if kind == "uniform" else init
    ex = _few_launches(off, idx, wt, init, most=40)
    assert ex.labels[1] == 0
    with R.Context(0) as ctx:
        r = ctx.refine(off, idx, wt, init)
        ctx.set_opts(verify=False)
        assert r.kernel_launches == ctx.refine(off, idx, wt, init).kernel_launches + 3


def test_long_member_of_few_colours_beside_short_rows():
    """60,000 arcs of the member read once for each of 5,000 rows."""
    n_short, k, heads = 5000, 60000, 1500
    src = np.concatenate([np.zeros(k + 1, np.int64), np.arange(1, n_short + 1)])
    dst = np.concatenate([n_short + 1 + np.arange(k) % heads, np.full(n_short + 1, n_short + 1 + heads)])
    n = n_short + heads + 2
    off, idx, w = G.csr_from_arcs(n, src, dst, np.where(dst == n - 1, 5, 0), sort=False)
    init = np.concatenate([np.zeros(n_short + 1), np.arange(1, heads + 2)]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, w, init)
    assert (ex.labels[: n_short + 1] == 0).all()
    with R.Context(0) as ctx:
        for _ in range(2):
            r = ctx.refine(off, idx, w, init)
            _same(r, ex)
            assert r.kernel_launches > 30  # decided launch by launch


def test_edge_batches_with_wide_rows():
    off, idx, init = _hubs(3000, 2, 2)
    off, idx = _marked(off, idx, init, 4, 4500)
    with R.Context(0) as ctx, R.Context(0, persistent=False) as per_phase:
        a, b = ctx.refine_edge_batches(off, idx)[0], per_phase.refine_edge_batches(off, idx)[0]
    assert a.blocks == b.blocks and np.array_equal(a.labels, b.labels)
    assert len(np.unique(a.labels[:4])) == 2
