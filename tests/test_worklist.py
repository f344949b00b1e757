"""The work list of deep refinements (deep_kernels.cuh) on classes that shed one
node per pass by a change of all their other nodes: the others move to a new
class id each time, so that such a class of s nodes uses about s ids, and a
graph of them more than half as many as it has nodes."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G


def shedding(length, groups, weighted=False):
    """Paths a, a', b (arcs j -> j - 1) coloured by position, with only b's first
    node told apart: b leaves the others one position per pass.  Node i of a
    group points at the first i nodes of b and the other nodes of a."""
    j = np.arange(1, length)
    src = [p * length + j for p in range(3)]
    dst = [p * length + j - 1 for p in range(3)]
    init = [np.arange(length), np.arange(length), np.concatenate([[length], np.arange(1, length)])]
    i, t = np.divmod(np.arange(length * length), length)
    for g in range(groups):
        src.append((3 + g) * length + i)
        dst.append(np.where(t < i, 2 * length + t, t))
        init.append(np.full(length, length + 1 + g))
    src, dst, init = np.concatenate(src), np.concatenate(dst), np.concatenate(init).astype(np.uint32)
    n = (3 + groups) * length
    perm = np.random.default_rng(length).permutation(n)
    off, idx, wt = G.csr_from_arcs(n, perm[src], perm[dst], np.full(len(src), 3) if weighted else None)
    out = np.empty(n, np.uint32)
    out[perm] = init
    return off, idx, wt, out


def _terms(c):
    x = (c.astype(np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
    x ^= x >> np.uint64(29)
    x *= np.uint64(0xBF58476D1CE4E5B9)
    return x ^ (x >> np.uint64(32))


def _ids_used(off, idx, init, full_passes):
    """The new class ids that the work list's rules hand out after so many full
    passes (a class of one node gets none), and the passes in all."""
    n = len(off) - 1
    off = off.astype(np.int64)
    sums = lambda c: np.concatenate([[np.uint64(0)], np.cumsum(_terms(c)[idx], dtype=np.uint64)])
    row = lambda c: (lambda s: s[off[1:]] - s[off[:-1]])(sums(c))
    col = np.unique(init, return_inverse=True)[1]
    for _ in range(full_passes):
        old = col
        col = np.unique(np.stack([col.astype(np.uint64), row(col)]), axis=1, return_inverse=True)[1].reshape(-1)
    # moved: not in the largest part of the class before
    part = np.bincount(col)[col]
    best = np.zeros(old.max() + 1, np.int64)
    np.maximum.at(best, old, part * (1 << 32) + col)
    moved = best[old] % (1 << 32) != col
    nid = first = col.max() + 1
    single = np.bincount(col, minlength=nid)[col] == 1
    passes = full_passes
    preds = lambda m: np.flatnonzero(np.add.reduceat(np.append(m[idx], 0), off[:-1]) * (np.diff(off) > 0))
    t = preds(moved)
    sig = row(col)
    base = {}
    rest = np.setdiff1d(np.arange(n), t)
    base.update(zip(col[rest].tolist(), sig[rest].tolist()))
    size = np.bincount(col).tolist()
    while True:
        groups = {}
        for u in t.tolist():
            if not single[u] and base.get(int(col[u])) != int(sig[u]):
                groups.setdefault(int(col[u]), {}).setdefault(int(sig[u]), []).append(u)
        moved = np.zeros(n, np.int64)
        new = 0
        for c, by_sum in groups.items():
            left = size[c] - sum(map(len, by_sum.values()))
            keeps = None if left else max(by_sum, key=lambda k: len(by_sum[k]))
            size[c] = left or len(by_sum[keeps])
            for s, us in by_sum.items():
                if s == keeps:
                    base[c] = s
                    continue
                new += 1
                moved[us] = 1
                if len(us) == 1:
                    single[us] = True
                    col[us[0]] = (1 << 31) | us[0]
                else:
                    col[us], base[nid] = nid, s
                    size.append(len(us))
                    nid += 1
        passes += 1
        if not new:
            return nid - first, passes
        t, sig = preds(moved), row(col)


SHAPES = [(60, 30, 10), (200, 10, 17)]  # length, groups, full passes before the work list


@pytest.mark.parametrize("length,groups,full", SHAPES)
def test_more_ids_than_half_the_nodes(length, groups, full):
    off, idx, _, init = shedding(length, groups)
    n = len(off) - 1
    ids, passes = _ids_used(off, idx, init, full)
    assert n // 2 + 2 < ids < n
    assert passes == oracle.refine_exact(off, idx, None, init).rounds


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("length,groups", [s[:2] for s in SHAPES] + [(64, 170)])
def test_classes_that_shed_nodes(length, groups, weighted):
    off, idx, wt, init = shedding(length, groups, weighted)
    ex = oracle.refine_exact(off, idx, wt, init)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx, wt)
        for r in (ctx.refine(off, idx, wt, init), g.refine(init), g.refine(init)):
            assert r.kernel_launches > 5  # the work list ran
            assert r.verified == 1 and (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
            assert np.array_equal(r.labels, ex.labels) and r.round_blocks == ex.round_blocks[: len(r.round_blocks)]
        g.free()


@pytest.mark.gpu
def test_the_last_allowed_pass_changes_many_sums():
    """3,000 nodes point at the first two nodes of a chain, which part last: more
    changed sums than the list holds, in the last pass but one."""
    length, many = 100, 3000
    c = np.arange(length - 1)
    p = length + np.arange(many)
    off, idx, _ = G.csr_from_arcs(length + many, np.concatenate([c, p, p]), np.concatenate([c + 1, 0 * p, 0 * p + 1]))
    init = np.concatenate([np.zeros(length), np.ones(many)]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    assert ex.rounds == length
    with R.Context(0, max_rounds=ex.rounds - 1) as ctx:
        with pytest.raises(R.RbscError, match="no fixpoint"):
            ctx.refine(off, idx, None, init)
        ctx.set_opts(max_rounds=ex.rounds)
        r = ctx.refine(off, idx, None, init)
        assert r.kernel_launches > 5 and r.verified == 1
        assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds) and np.array_equal(r.labels, ex.labels)
