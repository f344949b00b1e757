"""The one-launch refinement of small graphs (fused_kernels.cuh): labels, block
counts and rounds must equal the oracle's and the launch-per-phase path's, at
the sizes where its paths change (lane / group / warp / chunk rows, the check's
register and shared-memory rows, one cluster / whole chip)."""
import numpy as np
import pytest

import rbsc_b200 as R
from oracle import oracle
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu


def _twins(d, seed, n=3000):
    """Rows of exactly d arcs, each shared by four nodes: the twins stay in one
    block, so the exact check compares rows of d arcs."""
    rng = np.random.default_rng(seed)
    rows = [rng.integers(0, n, size=d) for _ in range(6)]
    src = np.concatenate([np.full(d, 4 * r + t) for r in range(6) for t in range(4)])
    dst = np.concatenate([rng.permutation(rows[r]) for r in range(6) for t in range(4)])
    tail = np.arange(24, n - 1)
    return G.csr_from_arcs(n, np.concatenate([src, tail]), np.concatenate([dst, tail + 1]), sort=False)[:2]


def _same(r, ex):
    assert r.done == 1 and r.verified == 1
    assert (r.blocks, r.rounds) == (ex.blocks, ex.rounds)
    assert np.array_equal(r.labels, ex.labels)
    assert r.round_blocks == ex.round_blocks[: len(r.round_blocks)]


def _both(off, idx, wt=None, init=None):
    ex = oracle.refine_exact(off, idx, wt, init)
    with R.Context(0) as ctx:
        one = ctx.refine(off, idx, wt, init)
        g = ctx.upload(off, idx, wt)
        a, b = g.refine(init), g.refine(init)
        g.free()
        ctx.set_opts(persistent=False)  # launch per phase
        slow = ctx.refine(off, idx, wt, init)
    for r in (one, a, b, slow):
        _same(r, ex)
    assert one.kernel_launches <= 2 < slow.kernel_launches
    return ex


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("d", [1, 8, 9, 12, 13, 16, 17, 32, 33, 128, 129, 192, 193, 512, 513, 1025])
def test_row_lengths(d, weighted):
    off, idx = _twins(d, seed=d)
    init = np.random.default_rng(d).integers(0, 40, size=len(off) - 1).astype(np.uint32)
    # rows of one colour multiset have equal weights only if the weights follow the heads
    wt = (idx.astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15) >> np.uint64(61)) + np.uint64(1) if weighted else None
    _both(off, idx, wt, init)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1025, 16384, 16385, 40000])
def test_node_counts(n):
    rng = np.random.default_rng(n)
    m = 3 * n
    off, idx, _ = G.csr_from_arcs(n, rng.integers(0, n, m), rng.integers(0, max(1, n // 3), m))
    _both(off, idx)
    _both(off, idx, None, R.degree_bucket_colors(off))


@pytest.mark.parametrize("n,m", [(900, 8191), (900, 8192), (900, 8193), (1024, 3000), (1025, 3000), (8192, (1 << 15) - 1),
                                 (8192, 1 << 15), (8193, 1 << 15), (8192, (1 << 15) + 1)])
def test_sizes_around_one_block_and_one_cluster(n, m):
    off, idx = G.er_directed(n, m, seed=m & 7)
    _both(off, idx, _rng_weights(m), None)
    _both(off, idx, None, (np.arange(n) % 9).astype(np.uint32))


def _rng_weights(m):
    return np.random.default_rng(m).integers(0, 3, size=m).astype(np.uint64)  # some weights are 0


@pytest.mark.parametrize("m", [(1 << 22) - 1, 1 << 22])
def test_largest_graphs(m):
    off, idx = G.er_directed(400000, m, seed=5)
    ex = oracle.refine_exact(off, idx)
    with R.Context(0) as ctx:
        r = ctx.refine(off, idx)
    _same(r, ex)
    assert (r.kernel_launches <= 2) == (m < 1 << 22)


def test_no_arcs_and_one_hub():
    _both(np.zeros(51, np.uint64), np.zeros(0, np.uint32), None, (np.arange(50) % 7).astype(np.uint32))
    off, idx = G.star_out(60000)  # one row of 59,999 arcs: over a hundred chunks
    _both(off, idx)


def test_row_wider_than_the_check_table():
    """Two nodes with the same 20,000 differently coloured heads: more colours
    than the check's table holds, so the call ends on the launch-per-phase path."""
    k = 20000
    heads = np.arange(2, k + 2)
    off, idx, _ = G.csr_from_arcs(k + 2, np.repeat([0, 1], k), np.tile(heads, 2))
    init = np.concatenate([[0, 0], heads]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0) as ctx:
        _same(ctx.refine(off, idx, None, init), ex)
        g = ctx.upload(off, idx)
        _same(g.refine(init), ex)
        g.free()


def test_row_wider_than_the_shared_table_without_allocation():
    """The same on rbsc_refine_noalloc, which counts such a row in its scratch."""
    import ctypes
    import torch
    from rbsc_b200 import _lib
    k = 6000
    heads = np.arange(3, k + 3)
    off, idx, _ = G.csr_from_arcs(k + 3, np.repeat([0, 1, 2], k), np.concatenate([heads, heads[::-1], heads % 5999 + 3]), sort=False)
    init = np.concatenate([[0, 0, 0], heads]).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    d = [torch.from_numpy(x).cuda() for x in (off.astype(np.int64), idx.view(np.int32), init.view(np.int32))]
    out, res = torch.zeros(k + 3, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    c = _lib.Csr()
    c.n, c.m, c.offsets, c.offset_bytes, c.indices, c.weights = k + 3, len(idx), d[0].data_ptr(), 8, d[1].data_ptr(), None
    o = _lib.Opts()
    _lib.load().rbsc_opts_default(ctypes.byref(o))
    for bits in (0, -1):  # -1: no signatures, every split comes from the exact check
        o.test_hash_bits = bits
        assert _lib.load().rbsc_refine_noalloc(ctypes.byref(c), d[2].data_ptr(), out.data_ptr(), res.data_ptr(), ctypes.byref(o), None) == 0
        torch.cuda.synchronize()
        assert res[3] == 0 and res[0] == ex.blocks and np.array_equal(out.cpu().numpy().view(np.uint32), ex.labels)


@pytest.mark.parametrize("bits", [2, -1])
@pytest.mark.parametrize("n,m", [(800, 3000), (20000, 70000)])
def test_collisions_are_repaired(bits, n, m):
    off, idx = G.er_directed(n, m, seed=4)
    init = (np.arange(n) % 3).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0, test_hash_bits=bits) as ctx:
        r = ctx.refine(off, idx, None, init)
    assert r.verified == 1 and r.blocks == ex.blocks and np.array_equal(r.labels, ex.labels)
    assert r.repairs > 0 or bits > 0  # two bits can still reach the fixpoint by themselves


@pytest.mark.parametrize("n", [500, 30000])
def test_errors_and_recovery(n):
    off, idx = G.er_directed(n, 4 * n, seed=8)
    off = off.astype(np.int64)
    bad_head = idx.copy()
    bad_head[n] = n
    dec = off.copy()
    dec[n // 2] = dec[n // 2 + 1] + 5
    first = off.copy()
    first[0] = 3
    with R.Context(0) as ctx:
        for o, i, text in ((off, bad_head, "head"), (dec, idx, "offsets"), (first, idx, "offsets")):
            with pytest.raises(R.RbscError, match=text):
                ctx.refine(o, i)
        ctx.set_opts(max_rounds=1)
        with pytest.raises(R.RbscError, match="no fixpoint"):
            ctx.refine(off, idx)
        ctx.set_opts(max_rounds=0)
        _same(ctx.refine(off, idx), oracle.refine_exact(off, idx))


def test_check_off_gives_the_same_labels():
    off, idx = G.random_lift(64, 400, 16, seed=3)
    ex = oracle.refine_exact(off, idx)
    with R.Context(0, verify=False) as ctx:
        r = ctx.refine(off, idx)
    assert r.verified == 0 and r.rounds == ex.rounds and np.array_equal(r.labels, ex.labels)


def test_device_pointers_and_small_offsets():
    """refine_device into a caller's tensor; 4-byte offsets give the same labels."""
    import torch
    off, idx = G.random_lift(700, 3000, 30, seed=6)
    init = (np.arange(len(off) - 1) % 5).astype(np.uint32)
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        d_init = torch.from_numpy(init.view(np.int32)).cuda()
        d_out = torch.full((g.n,), -1, dtype=torch.int32, device="cuda")
        r = g.refine_device(d_init.data_ptr(), d_out.data_ptr())
        assert r.blocks == ex.blocks and np.array_equal(d_out.cpu().numpy().view(np.uint32), ex.labels)
        g.free()
        _same(ctx.refine(off.astype(np.uint32), idx, None, init), ex)


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("chain", [40, 64, 65, 700])
@pytest.mark.parametrize("nodes", [3, 300])
def test_many_rounds(nodes, chain, weighted):
    """Enough passes for the work-list tail: a chain beside a lift whose blocks
    keep several nodes (chains hang off every copy, so whole blocks move)."""
    lift = 6
    off, idx = G.random_lift(nodes, 2 * nodes, lift, seed=chain)
    n = len(off) - 1
    s, d = G.arcs_of(off, idx)
    k = np.arange(chain - 1)
    src, dst = [s, np.arange(lift)], [d, np.full(lift, n)]  # the copies of base node 0 point at the chain
    for c in range(3):  # three equal chains: their nodes share blocks
        src.append(n + c * chain + k)
        dst.append(n + c * chain + k + 1)
    src, dst = np.concatenate(src), np.concatenate(dst)
    perm = np.random.default_rng(chain).permutation(n + 3 * chain)
    off2, idx2, wt2 = G.csr_from_arcs(n + 3 * chain, perm[src], perm[dst], np.full(len(src), 3) if weighted else None)
    ex = oracle.refine_exact(off2, idx2, wt2)
    assert ex.rounds >= chain // 2
    with R.Context(0) as ctx:
        for _ in range(2):
            _same(ctx.refine(off2, idx2, wt2), ex)
        g = ctx.upload(off2, idx2, wt2)
        _same(g.refine(), ex)
        g.free()
        ctx.set_opts(max_rounds=ex.rounds - 1)
        with pytest.raises(R.RbscError, match="no fixpoint"):
            ctx.refine(off2, idx2, wt2)
        ctx.set_opts(max_rounds=ex.rounds)
        _same(ctx.refine(off2, idx2, wt2), ex)


def test_many_rounds_with_wide_passes():
    """Passes that change more sums than the work list holds go back to full
    passes: 1,500 chains of 60 nodes, each node pointed at by two more."""
    c, k = 1500, 60
    base = np.arange(c * k).reshape(c, k)
    src = np.concatenate([base[:, :-1].ravel(), c * k + base.ravel(), 2 * c * k + base.ravel()])
    dst = np.concatenate([base[:, 1:].ravel(), base.ravel(), base.ravel()])
    init = np.zeros(3 * c * k, np.uint32)
    off, idx, _ = G.csr_from_arcs(3 * c * k, src, dst)
    ex = oracle.refine_exact(off, idx, None, init)
    assert ex.rounds >= 55
    with R.Context(0) as ctx:
        _same(ctx.refine(off, idx, None, init), ex)


@pytest.mark.parametrize("n", [1, 2, 40, 1025, 6000])
def test_paths_and_cycles(n):
    for off, idx in ((G.path(n), G.cycle(n)) if n > 1 else (G.cycle(n),)):
        with R.Context(0) as ctx:
            _same(ctx.refine(off, idx), oracle.refine_exact(off, idx))


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("m", [(1 << 22) + 7, 3 << 23])
def test_large_resident_graphs(m, weighted):
    """From 2^22 arcs on one launch takes a resident graph with no initial
    colours (to 24 M arcs, weighted to 32 M), with the other path's result."""
    off, idx = R.gen_er_host(600000, m / 600000, seed=m & 63)
    wt = np.random.default_rng(1).integers(0, 4, size=len(idx)).astype(np.uint64) if weighted else None
    with R.Context(0) as ctx, R.Context(0, persistent=False) as per_phase:
        for init in (None, R.degree_bucket_colors(off)):
            g = ctx.upload(off, idx, wt)
            a = g.refine(init)
            g.free()
            b = per_phase.refine(off, idx, wt, init)
            assert (a.blocks, a.rounds, a.round_blocks) == (b.blocks, b.rounds, b.round_blocks)
            assert np.array_equal(a.labels, b.labels) and a.verified == b.verified == 1
            if init is None:
                assert (a.kernel_launches <= 2) == (len(idx) < (1 << 25 if weighted else 3 << 23))


def _wide(k):
    heads = np.arange(2, k + 2)
    off, idx, _ = G.csr_from_arcs(k + 2, np.repeat([0, 1], k), np.tile(heads, 2))
    return off, idx, np.concatenate([[0, 0], heads]).astype(np.uint32)


@pytest.mark.parametrize("kind", ["block", "cluster", "grid", "deep", "wide", "large"])
def test_labels_over_the_initial_colours(kind):
    """The label array may be the array of the initial colours."""
    import ctypes
    import torch
    from rbsc_b200 import _lib
    if kind == "wide":
        off, idx, init = _wide(20000)  # starts again launch by launch
    else:
        if kind == "deep":
            off, idx = G.random_lift(300, 600, 6, seed=1)
            s, d = G.arcs_of(off, idx)
            n, k = len(off) - 1, np.arange(300)
            off, idx, _ = G.csr_from_arcs(n + 301, np.concatenate([s, n + k]), np.concatenate([d, n + k + 1]))
        else:
            nodes, lift = dict(block=(40, 8), cluster=(600, 12), grid=(4000, 16), large=(20000, 32))[kind]
            off, idx = G.random_lift(nodes, nodes * 7, lift, seed=1)
        init = (np.arange(len(off) - 1) % 3).astype(np.uint32)
        init[: len(init) // 2] = 5  # rows of one colour that stay together, of several that do not
    n = len(off) - 1
    ex = oracle.refine_exact(off, idx, None, init)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        buf = torch.from_numpy(init.view(np.int32)).cuda()
        r = g.refine_device(buf.data_ptr(), buf.data_ptr())
        assert r.blocks == ex.blocks and np.array_equal(buf.cpu().numpy().view(np.uint32), ex.labels)
        g.free()
    if n <= 16384 and len(idx) <= 1 << 16:
        d = [torch.from_numpy(x).cuda() for x in (off.astype(np.int64), idx.view(np.int32), init.view(np.int32))]
        res = torch.zeros(4, dtype=torch.int32, device="cuda")
        c = _lib.Csr()
        c.n, c.m, c.offsets, c.offset_bytes, c.indices, c.weights = n, len(idx), d[0].data_ptr(), 8, d[1].data_ptr(), None
        torch.cuda.synchronize()
        assert _lib.load().rbsc_refine_noalloc(ctypes.byref(c), d[2].data_ptr(), d[2].data_ptr(), res.data_ptr(), None, None) == 0
        torch.cuda.synchronize()
        assert res[3] == 0 and np.array_equal(d[2].cpu().numpy().view(np.uint32), ex.labels)
