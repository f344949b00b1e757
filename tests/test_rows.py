"""The later passes of a large refinement in one launch (list_kernels.cuh):
labels, block counts and rounds must equal the oracle's and the
launch-per-phase path's, for each kind of first pass and at the row lengths
where the pass's and the check's ways part."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu

HEADS = 3000  # nodes of the special part, before the filler


@pytest.fixture(scope="module")
def filler():
    """Enough arcs for the path: 2^22 from 150,000 nodes, and 20,000 nodes without arcs."""
    rng = np.random.default_rng(12)
    m, n = 1 << 22, 150000
    return n + 20000, np.sort(rng.integers(0, n, size=m)), rng.integers(0, n + 20000, size=m)


def _with(filler, src, dst, heads=HEADS):
    n, fs, fd = filler
    return G.csr_from_arcs(heads + n, np.concatenate([src, fs + heads]), np.concatenate([dst, fd + heads]), sort=False)[:2]


def _same(r, ex):
    assert r.done == 1 and r.verified == 1
    assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
    assert np.array_equal(r.labels, ex.labels)
    assert r.round_blocks == ex.round_blocks[: len(r.round_blocks)]


def _check(off, idx, init, rows=True):
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0) as ctx:
        one = ctx.refine(off, idx, None, init)
        g = ctx.upload(off, idx)
        a, b = g.refine(init), g.refine(init)
        ctx.set_opts(persistent=False)  # launch per phase
        slow = g.refine(init)
        ctx.set_opts(persistent=True)
        c = g.refine(init)
        g.free()
    for r in (one, a, b, slow, c):
        _same(r, ex)
    if rows:
        assert c.kernel_launches < slow.kernel_launches
    return ex


@pytest.mark.parametrize("d", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 1025])
def test_row_lengths(filler, d):
    """Six times four rows of d arcs over the same heads, in any order."""
    rng = np.random.default_rng(d)
    rows = [rng.integers(24, HEADS, size=d) for _ in range(6)]
    src = np.concatenate([np.full(d, 4 * r + t) for r in range(6) for t in range(4)])
    dst = np.concatenate([rng.permutation(rows[r]) for r in range(6) for t in range(4)])
    off, idx = _with(filler, src, dst)
    init = rng.integers(0, 3, size=len(off) - 1).astype(np.uint32)
    init[:24] = 1
    ex = _check(off, idx, init)
    assert len(np.unique(ex.labels[:24])) <= 6


@pytest.mark.parametrize("classes", [1, 200, 5000, 100000], ids=["one", "rank8", "rank16", "full"])
def test_first_passes(filler, classes):
    rng = np.random.default_rng(classes)
    tail = np.arange(HEADS - 1)
    off, idx = _with(filler, tail[:7], tail[:7] + 1)
    init = None if classes == 1 else rng.integers(0, classes, size=len(off) - 1).astype(np.uint32)
    _check(off, idx, init, rows=init is not None)  # (a resident one-class graph of this size is one launch as a whole)


def test_a_row_wider_than_the_check_table_ends_launch_by_launch(filler):
    k = 5000
    heads = np.arange(2, k + 2)
    off, idx = _with(filler, np.repeat([0, 1], k), np.concatenate([heads, heads[::-1]]), heads=k + 2)
    init = np.zeros(len(off) - 1, dtype=np.uint32)
    init[2:k + 2] = heads
    _check(off, idx, init, rows=False)


def test_errors_and_recovery(filler):
    off, idx = _with(filler, [0], [1])
    init = R.degree_bucket_colors(off)
    bad = idx.copy()
    bad[len(bad) // 2] = len(off) - 1
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0) as ctx:
        with pytest.raises(R.RbscError, match="head"):
            ctx.refine(off, bad, None, init)
        g = ctx.upload(off, idx)
        ctx.set_opts(max_rounds=1)
        with pytest.raises(R.RbscError, match="no fixpoint"):
            g.refine(init)
        ctx.set_opts(max_rounds=0)
        _same(g.refine(init), ex)
        ctx.set_opts(verify=False)
        r = g.refine(init)
        assert r.verified == 0 and np.array_equal(r.labels, ex.labels)
        g.free()


def test_many_refinements_of_one_graph(filler):
    """One stamp of the initial colours' table a refinement: 255 fill its turn."""
    off, idx = _with(filler, [0], [1])
    init = R.degree_bucket_colors(off)
    other = (init * 3 + np.arange(len(init), dtype=np.uint32) % 2).astype(np.uint32)
    want = [oracle.refine_exact(off, idx, None, i) for i in (init, other)]
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        for k in range(520):
            r, ex = g.refine((init, other)[k % 2]), want[k % 2]
            assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds), k
            assert np.array_equal(r.labels, ex.labels), k
        g.free()
