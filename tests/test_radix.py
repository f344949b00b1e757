"""The radix sort (radix.cuh) through the entry points that sort: the edges of
its 4,096-key tiles, digits that end inside a byte, values of 4 and 8 bytes."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 4095, 4096, 4097, 12289, 200001])
def test_sort_relabel(n):
    """32-, 64- and 31-bit sorts of n keys with 4-byte values; every pass sorts."""
    rng = np.random.default_rng(n)
    m = 2 * n
    off, idx, _ = G.csr_from_arcs(n, rng.integers(0, n, m), rng.integers(0, max(1, n // 2), m))
    init = rng.integers(0, 3, n).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0, relabel=R.RELABEL_SORT) as ctx:
        r = ctx.refine(off, idx, None, init)
    assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds) and np.array_equal(r.labels, ex.labels)


@pytest.mark.parametrize("scale", [10, 13, 17])
def test_generator_sorts_like_the_host(scale):
    """Keys without values, 2 * scale bits (a last digit of 2, 4 and 2 bits)."""
    off, idx = R.gen_rmat_host(scale, 9, seed=scale)
    with R.Context(0) as ctx:
        g = ctx.gen_rmat_pinned(scale, 9, seed=scale)
        assert np.array_equal(g.off, off) and np.array_equal(g.idx, idx)
        g.free()


@pytest.mark.parametrize("n,m", [(40, 4096), (3000, 4097), (70000, 300000)])
def test_double_weights(n, m):
    """8-byte values in arc order inside equal keys (the order of the sums), and
    the check's sort with 4-byte values."""
    rng = np.random.default_rng(m)
    off, idx, _ = G.csr_from_arcs(n, rng.integers(0, n, m), rng.integers(0, n, m))
    wt = rng.choice([0.1, 0.2, 0.3, 1e-9, 7.0, -0.3], size=len(idx))
    ex = oracle.refine_f64(off, idx, wt)
    with R.Context(0) as ctx:
        r = ctx.refine_f64(off, idx, wt)
    assert r.blocks == ex.blocks and np.array_equal(r.labels, ex.labels)


def test_long_rows_of_the_check():
    """Rows of more than 32 arcs, unit and weighted, sorted by the check of the
    launch-per-phase path."""
    off, idx = G.random_lift(60, 60 * 45, 8, seed=2)
    for wt in (None, (idx % 3 + 1).astype(np.uint64)):
        ex = oracle.refine_exact(off, idx, wt)
        with R.Context(0, persistent=False) as ctx:
            r = ctx.refine(off, idx, wt)
        assert r.blocks == ex.blocks and np.array_equal(r.labels, ex.labels) and r.verified == 1


@pytest.mark.parametrize("n_rows", [1, 3])
@pytest.mark.parametrize("d", [32, 33, 127, 128, 129, 256, 257, 5000])
def test_long_groups_of_double_weights(d, n_rows):
    """Rows of d arcs into one block, summed in arc order (the float of the sum
    depends on it); rows that end up alone leave the later passes."""
    rng = np.random.default_rng(d)
    n = 600
    src = np.concatenate([np.repeat(np.arange(2 * n_rows), d), np.arange(50, n - 1)])
    dst = np.concatenate([rng.integers(300, n, 2 * n_rows * d), np.arange(51, n)])
    w = rng.choice([0.1, 1e8, -1e8, 3e-5, 0.7], size=n_rows * d)
    wt = np.concatenate([w, w, np.full(n - 51, 0.3)])  # the second half repeats the first: equal rows
    dst[n_rows * d: 2 * n_rows * d] = dst[: n_rows * d]
    off, idx, order = G.csr_from_arcs(n, src, dst, np.arange(len(src)), sort=False)
    wt = wt[order.astype(np.int64)]
    ex = oracle.refine_f64(off, idx, wt)
    with R.Context(0) as ctx:
        r = ctx.refine_f64(off, idx, wt)
    assert r.blocks == ex.blocks and np.array_equal(r.labels, ex.labels) and r.rounds == ex.rounds
