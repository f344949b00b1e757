"""Which way a sparse graph of many nodes takes, and that it gives the oracle's
result there."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


def _er(n, m, seed):
    rng = np.random.default_rng(seed)
    src = np.sort(rng.integers(0, n, m))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint64)
    return off, rng.integers(0, n, m).astype(np.uint32)


def _same(r, ex):
    assert r.done == 1 and r.verified == 1
    assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
    assert np.array_equal(r.labels, ex.labels)


@pytest.mark.parametrize("seed", [1, 2])
def test_passes_that_soon_make_no_more_classes(seed):
    """A random graph's last passes make fewer and fewer classes: no work list for
    the one or two that are left."""
    off, idx = _er(1 << 20, 734003, seed)
    ex = oracle.refine_exact(off, idx)
    assert ex.rounds >= 15
    with R.Context(0) as ctx:
        r = ctx.refine(off, idx)
    _same(r, ex)
    assert r.kernel_launches <= 2


@pytest.mark.parametrize("chain,extra", [(60, 0), (400, 0), (60, 300)])
def test_passes_that_go_on_making_classes(chain, extra):
    """Chains keep making the same number: the work list takes over, also after
    passes that made many at once (extra: nodes with rows of their own)."""
    k = np.arange(chain)
    src, dst = [k, 20000 + k], [k + 1, 20000 + k + 1]
    n = 40000
    for e in range(extra):
        src.append(np.full(e % 7 + 1, 30000 + e))
        dst.append(30000 + (e * 13 + np.arange(e % 7 + 1)) % 301)
    off, idx, _ = G.csr_from_arcs(n, np.concatenate(src), np.concatenate(dst))
    ex = oracle.refine_exact(off, idx)
    with R.Context(0) as ctx:
        r = ctx.refine(off, idx)
    _same(r, ex)
    assert r.rounds > chain and r.kernel_launches > 5


def test_passes_that_make_more_and_fewer_classes_in_turn():
    """A chain, and at every other node of it five nodes, each of a colour with one
    at the first: they part when that node does, 6, 1, 6, 1 new classes."""
    chain, each = 300, 5
    k = np.arange(chain)
    at = np.repeat(np.arange(0, chain, 2), each)
    x = chain + 1 + 2 * np.arange(len(at))
    n = chain + 1 + 2 * len(at)
    off, idx, _ = G.csr_from_arcs(n, np.concatenate([k, x, x + 1]), np.concatenate([k + 1, at, 0 * at]))
    init = np.concatenate([np.zeros(chain + 1), 1 + np.arange(2 * len(at)) // 2]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    new = np.diff(ex.round_blocks[20:280])
    assert set(new) == {1, 1 + each}
    with R.Context(0) as ctx:
        r = ctx.refine(off, idx, None, init)
    _same(r, ex)
    assert r.kernel_launches > 5


@pytest.mark.parametrize("n,m,phases", [(1 << 20, 1 << 19, False), ((1 << 20) + 1, 1 << 19, True), ((1 << 20) + 8, (1 << 20) + 9 + (1 << 17), False),
                                        ((1 << 20) + 8, (1 << 20) + 8 + (1 << 17), True), ((1 << 22) - 7, 90001, True)])
def test_sparse_graphs_of_many_nodes(n, m, phases):
    """Resident and unweighted, launch by launch; in one launch otherwise."""
    off, idx = _er(n, m, 3)
    ex = oracle.refine_exact(off, idx)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        for _ in range(2):
            r = g.refine()
            _same(r, ex)
            assert (r.kernel_launches > 5) == phases
        g.free()
        r = ctx.refine(off, idx)
        _same(r, ex)
        assert r.kernel_launches <= 2
        wt = np.full(m, 3, np.uint64)
        g = ctx.upload(off, idx, wt)
        r = g.refine()
        _same(r, oracle.refine_exact(off, idx, wt))
        assert r.kernel_launches <= 2
        g.free()
