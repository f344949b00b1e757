"""The workloads this library's speed is judged on: graphs, entry points and
sizes as users of the library call it.

A case names an entry point (`call`), a graph (`graph` and its sizes) and the
options of the call.  Graph families:

    rmat    directed R-MAT, 2^scale nodes, edge_factor * 2^scale generated arcs
            (skewed in- and out-degrees, as web and social graphs)
    er      directed Erdos-Renyi of `nodes` nodes and `degree` mean out-degree
    lift    random lift of an Erdos-Renyi base: `nodes` base nodes, each copied
            `lift` times (many nodes per block at the fixpoint), node ids shuffled
    deep    a lift beside a path of `chain` nodes: about `chain` rounds, as a web
            crawl's long chains give (the reference's cnr-2000 sample needs 173)
    wl      `graphs` small graphs, half Erdos-Renyi and half 3-regular, labels
            1..8 (the 1-WL expressiveness sweep), each graph's node ids shuffled
    mix     `jobs` graphs of log-uniform size, lift / rmat / er in turn (the
            served request mix)

Initial colours: none (one block) or floor(log2(out-degree + 1)).
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

import rbsc_b200 as R
from rbsc_b200 import _lib


def listed():
    return [
        # plain refinement at scale: a graph kept in device memory and refined
        # again and again from degree colours (the headline workload)
        dict(name="resident_rmat24", call="resident", graph="rmat", scale=24, edge_factor=16, init="degree", weighted=False),
        # plain refinement, small: the 131,072-node random lift, one initial block
        dict(name="resident_lift131k", call="resident", graph="lift", nodes=4096, degree=8.0, lift=32, init="none",
             weighted=False),
        # weighted lumping: integer arc weights on a skewed graph
        dict(name="resident_weighted_rmat20", call="resident", graph="rmat", scale=20, edge_factor=16, init="none",
             weighted=True),
        # many rounds over a small graph: the size and depth of a web crawl
        # sample (cnr-2000: 325,557 nodes, 3.2 M arcs, 173 rounds)
        dict(name="resident_deep320k", call="resident", graph="deep", nodes=10174, degree=9.9, lift=32, chain=170, init="none",
             weighted=False),
        # the smallest calls: one request of about a thousand arcs, host arrays in, labels out
        dict(name="oneshot_er1k", call="oneshot", graph="er", nodes=331, degree=3.0, init="none", weighted=False, pinned=False,
             offset_bytes=4),
        # one-shot refinement of a large graph from page-locked host arrays
        dict(name="oneshot_rmat22", call="oneshot", graph="rmat", scale=22, edge_factor=16, init="degree", weighted=False,
             pinned=True, offset_bytes=8),
        # the batched sweep: 100,000 small graphs in one call, per-graph results out
        dict(name="batch_100k", call="batch", graph="wl", graphs=100000, nmin=10, nmax=500, pinned=True),
        # the allocation-free entry point, on a caller's device arrays
        dict(name="noalloc_er5k", call="noalloc", graph="er", nodes=5003, degree=6.0, init="none", weighted=False,
             offset_bytes=8),
        # lumping with double weights
        dict(name="f64_rmat20", call="f64", graph="rmat", scale=20, edge_factor=16, init="none"),
        # the reference's edge-batch (quotient) mode, a quarter of the arcs per batch
        dict(name="edge_batches_rmat20", call="edge_batches", graph="rmat", scale=20, edge_factor=16, parts=4, aggressive=False),
        # arcs in host memory, streamed in quarters during the signature passes
        dict(name="streamed_rmat22", call="streamed", graph="rmat", scale=22, edge_factor=32, parts=4, init="degree"),
        # the service: a burst of requests of mixed sizes through one server
        dict(name="served_mix32", call="served", graph="mix", jobs=32, arcs_lo=1000, arcs_hi=4000000),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _logi(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def _er(rng, lo, hi):
    # sparse enough that some nodes share a block
    n = _logi(rng, lo, hi)
    return dict(nodes=n, degree=round(rng.uniform(1.3, min(10.0, np.log(n) - 1.5)), 2))


def draw(rng):
    call = rng.choice(["resident", "resident", "resident", "oneshot", "oneshot", "batch", "noalloc", "f64", "edge_batches",
                       "streamed", "served"])
    if call == "batch":
        nmin = rng.randint(5, 40)
        return dict(call=call, graph="wl", graphs=_logi(rng, 50, 90000), nmin=nmin, nmax=nmin + rng.randint(20, 460),
                    pinned=rng.random() < 0.5)
    if call == "served":
        return dict(call=call, graph="mix", jobs=rng.randint(8, 48), arcs_lo=1000, arcs_hi=_logi(rng, 20000, 3000000))
    if call == "noalloc":
        return dict(call=call, graph="er", **_er(rng, 300, 16384), init=rng.choice(["none", "degree"]),
                    weighted=rng.random() < 0.3, offset_bytes=rng.choice([4, 8]))
    if call in ("f64", "edge_batches", "streamed"):
        c = dict(call=call, graph="rmat", scale=rng.randint(14, 20), edge_factor=rng.randint(5, 16))
        if call == "f64":
            c["init"] = rng.choice(["none", "degree"])
        else:
            c["parts"] = rng.randint(2, 6)
            if call == "edge_batches":
                c["aggressive"] = rng.random() < 0.3
            else:
                c["init"] = rng.choice(["none", "degree"])
        return c
    c = dict(call=call, init=rng.choice(["none", "degree"]), weighted=rng.random() < 0.25)
    c["graph"] = rng.choice(["rmat", "er", "lift"] + (["deep"] if call == "resident" else []))
    if c["graph"] == "rmat":
        c.update(scale=rng.randint(11, 20 if c["weighted"] else 22), edge_factor=rng.randint(5, 16))
    elif c["graph"] == "er":
        c.update(_er(rng, 300, 1500000))
    else:
        c.update(nodes=_logi(rng, 16, 20000 if c["graph"] == "lift" else 9000), degree=round(rng.uniform(2.0, 10.0), 2),
                 lift=rng.randint(2, 40))
        if c["graph"] == "deep":
            c.update(chain=_logi(rng, 20, 170), weighted=False)
    if call == "oneshot":
        c.update(pinned=rng.random() < 0.5, offset_bytes=rng.choice([4, 8]))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_ctx = None
_server = None


def _context():
    # a program keeps one context for all its graphs
    global _ctx
    if _ctx is None:
        _ctx = R.Context(torch.cuda.current_device())
    return _ctx


def _serving():
    global _server
    if _server is None:
        _server = R.Server(torch.cuda.current_device(), slots=2)
    return _server


def _relabel(off, idx, rank):
    """The graph with node u renamed to the position of rank[u] in sorted order
    (on the GPU: the batch has 25 M nodes)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    off = torch.from_numpy(off.astype(np.int64)).to(dev)
    idx = torch.from_numpy(idx.astype(np.int64)).to(dev)
    old = torch.argsort(torch.from_numpy(rank).to(dev))
    new = torch.empty_like(old)
    new[old] = torch.arange(old.numel(), device=dev)
    deg = (off[1:] - off[:-1])[old]
    noff = torch.zeros_like(off)
    torch.cumsum(deg, 0, out=noff[1:])
    src = torch.repeat_interleave(off[:-1][old] - noff[:-1], deg) + torch.arange(idx.numel(), device=dev)
    return noff.cpu().numpy().view(np.uint64), new[idx[src]].to(torch.int32).cpu().numpy().view(np.uint32)


def _lift(nodes, degree, lift, seed, chain=0):
    off, idx = R.gen_lift_host(nodes, degree, lift, seed=seed)
    if chain:
        n, m = len(off) - 1, len(idx)
        off = np.concatenate([off, m + np.minimum(np.arange(1, chain + 1), chain - 1).astype(np.uint64)])
        idx = np.concatenate([idx, (n + np.arange(1, chain)).astype(np.uint32)])
    return _relabel(off, idx, np.random.default_rng(seed + 79).random(len(off) - 1))


def _batch(case, seed):
    """The sweep's graphs side by side: sizes and shapes fixed by the case; node
    ids inside each graph and labels by the seed."""
    off, idx, gn, _ = R.gen_wl_batch(case["graphs"], case["nmin"], case["nmax"], seed=case["graphs"])
    n = len(off) - 1
    rng = np.random.default_rng(seed + 80)
    graph = np.repeat(np.arange(len(gn) - 1), np.diff(gn.astype(np.int64)))
    off, idx = _relabel(off, idx, graph + 0.999 * rng.random(n))
    return off, idx, gn, rng.integers(1, 9, size=n).astype(np.uint32)


def _host_graph(case, seed):
    """(offsets uint64, heads uint32) on the host."""
    kind = case["graph"]
    if kind == "rmat":
        if case["scale"] < 16:
            return R.gen_rmat_host(case["scale"], case["edge_factor"], seed=seed)
        g = _context().gen_rmat_pinned(case["scale"], case["edge_factor"], seed=seed)
        off, idx = g.off.copy(), g.idx.copy()
        g.free()
        return off, idx
    if kind == "er":
        return R.gen_er_host(case["nodes"], case["degree"], seed=seed)
    return _lift(case["nodes"], case["degree"], case["lift"], seed, case.get("chain", 0))


def _weights(m, seed):
    return np.random.default_rng(seed + 77).integers(1, 5, size=m).astype(np.uint64)


def _doubles(m, seed):
    # multiples of 1/2: rates as a model's author writes them
    return np.random.default_rng(seed + 78).integers(1, 9, size=m).astype(np.float64) * 0.5


def _init(case, off):
    return R.degree_bucket_colors(off) if case.get("init") == "degree" else None


def _pin(a):
    if a is None:
        return None
    a = np.ascontiguousarray(a)
    t = torch.empty(max(a.nbytes, 1), dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[: a.nbytes].view(a.dtype)
    v[:] = a
    return v


def _mix(case, seed):
    sizes = np.random.default_rng(case["jobs"])
    out = []
    for j in range(case["jobs"]):
        arcs = case["arcs_lo"] * (case["arcs_hi"] / case["arcs_lo"]) ** sizes.random()
        s = seed * 1000 + j
        if j % 3 == 0:
            out.append(_lift(max(2, int(arcs / 8 / 32)), 8.0, 32, s))
        elif j % 3 == 1:
            out.append(R.gen_rmat_host(max(5, int(np.log2(max(arcs / 16, 32)))), 16, seed=s))
        else:
            out.append(R.gen_er_host(max(8, int(arcs / 6)), 6.0, seed=s))
    return out


def prepare(case, seed):
    call = case["call"]
    st = dict(call=call)
    if call == "served":
        st.update(server=_serving(), jobs=_mix(case, seed))
        return st
    ctx = st["ctx"] = _context()
    if call == "batch":
        off, idx, gn, lab = _batch(case, seed)
        if case["pinned"]:
            off, idx, lab = _pin(off), _pin(idx), _pin(lab)
        # output arrays a program keeps from call to call
        st["out"] = R.batch_buffers(len(off) - 1, len(gn) - 1,
                                    alloc=lambda n, dt: _pin(np.zeros(n, dt)) if case["pinned"] else np.zeros(n, dt))
        st.update(off=off, idx=idx, gn=gn, init=lab)
        return st
    if call == "resident":
        if case["graph"] == "rmat" and not case["weighted"]:
            g = ctx.gen_rmat(case["scale"], case["edge_factor"], seed=seed)
            init = None
            if case["init"] == "degree":
                init = torch.empty(g.n, dtype=torch.int32, device="cuda")
                g.degree_colors_device(init.data_ptr())
        else:
            off, idx = _host_graph(case, seed)
            g = ctx.upload(off, idx, _weights(len(idx), seed) if case["weighted"] else None)
            init = _init(case, off)
            init = None if init is None else torch.from_numpy(init.view(np.int32)).cuda()
        st.update(g=g, init=init, labels=torch.empty(g.n, dtype=torch.int32, device="cuda"))
        return st
    if call == "streamed":
        pg = ctx.gen_rmat_pinned(case["scale"], case["edge_factor"], seed=seed)
        g = ctx.upload_streamed(pg.off, pg.idx, batch_arcs=max(1, pg.m // case["parts"]))
        init = None
        if case["init"] == "degree":
            init = torch.empty(g.n, dtype=torch.int32, device="cuda")
            g.degree_colors_device(init.data_ptr())
        st.update(pg=pg, g=g, init=init, labels=torch.empty(g.n, dtype=torch.int32, device="cuda"))
        return st
    off, idx = _host_graph(case, seed)
    if call == "f64":
        st.update(off=off, idx=idx, wt=_doubles(len(idx), seed), init=_init(case, off))
        return st
    if call == "edge_batches":
        st.update(off=off, idx=idx, size=max(1, -(-len(idx) // case["parts"])), aggressive=case["aggressive"])
        return st
    wt = _weights(len(idx), seed) if case["weighted"] else None
    init = _init(case, off)
    if call == "oneshot":
        off = off.astype(np.uint32) if case["offset_bytes"] == 4 else off
        out = None
        if case["pinned"]:
            off, idx, wt, init = _pin(off), _pin(idx), _pin(wt), _pin(init)
            out = _pin(np.zeros(len(off) - 1, np.uint32))
        st.update(off=off, idx=idx, wt=wt, init=init, out=out)
        return st
    # noalloc: the caller's own device arrays
    n = len(off) - 1
    d = dict(off=torch.from_numpy(off.astype(np.int64 if case["offset_bytes"] == 8 else np.int32)).cuda(),
             idx=torch.from_numpy(idx.view(np.int32)).cuda(),
             wt=None if wt is None else torch.from_numpy(wt.view(np.int64)).cuda(),
             init=None if init is None else torch.from_numpy(init.view(np.int32)).cuda(),
             out=torch.empty(n, dtype=torch.int32, device="cuda"), res=torch.zeros(4, dtype=torch.int32, device="cuda"))
    c = _lib.Csr()
    c.n, c.m, c.offsets, c.offset_bytes = n, len(idx), d["off"].data_ptr(), case["offset_bytes"]
    c.indices = d["idx"].data_ptr() if len(idx) else None
    c.weights = d["wt"].data_ptr() if wt is not None else None
    st.update(d=d, csr=c, lib=_lib.load())
    return st


def run(st):
    call = st["call"]
    if call in ("resident", "streamed"):
        r = st["g"].refine_device(None if st["init"] is None else st["init"].data_ptr(), st["labels"].data_ptr())
        return dict(labels=st["labels"], blocks=r.blocks, rounds=r.rounds)
    if call == "oneshot":
        r = st["ctx"].refine(st["off"], st["idx"], st["wt"], st["init"], out=st["out"])
        return dict(labels=r.labels, blocks=r.blocks, rounds=r.rounds)
    if call == "batch":
        b = st["ctx"].batch_refine(st["off"], st["idx"], st["gn"], init=st["init"], out=st["out"])
        o = st["out"]
        return dict(colors=b.colors, local=b.local, per_graph=b.blocks, hist_offsets=b.hist_offsets, hist_colors=o["hist_colors"],
                    hist_counts=o["hist_counts"], fingerprint=b.fingerprint.view(np.int64), blocks=b.stats.blocks,
                    rounds=b.stats.rounds)
    if call == "noalloc":
        d = st["d"]
        s = st["lib"].rbsc_refine_noalloc(ctypes.byref(st["csr"]), None if d["init"] is None else d["init"].data_ptr(),
                                          d["out"].data_ptr(), d["res"].data_ptr(), None,
                                          torch.cuda.current_stream().cuda_stream)
        return dict(labels=d["out"], result=d["res"], status=s)
    if call == "f64":
        r = st["ctx"].refine_f64(st["off"], st["idx"], st["wt"], st["init"])
        return dict(labels=r.labels, blocks=r.blocks, rounds=r.rounds)
    if call == "edge_batches":
        r, info = st["ctx"].refine_edge_batches(st["off"], st["idx"], edge_batch_size=st["size"], aggressive=st["aggressive"])
        return dict(labels=r.labels, blocks=r.blocks, done=r.done, iterations=info["iterations"])
    ids = [st["server"].submit(off, idx) for off, idx in st["jobs"]]
    res = [st["server"].wait(i) for i in ids]
    return dict(labels=[r.labels for r in res], blocks=np.array([r.blocks for r in res], dtype=np.int64))


# ---------------------------------------------------------------------------
# work and exact results
# ---------------------------------------------------------------------------
def _size(case):
    kind = case["graph"]
    if kind == "rmat":
        return 1 << case["scale"], case["edge_factor"] << case["scale"]
    if kind == "er":
        return case["nodes"], int(case["nodes"] * case["degree"])
    if kind in ("lift", "deep"):
        n = case["nodes"] * case["lift"] + case.get("chain", 0)
        return n, int(case["nodes"] * case["lift"] * case["degree"]) + case.get("chain", 0)
    if kind == "wl":
        n = int(case["graphs"] * (case["nmin"] + case["nmax"]) / 2)
        return n, int(3.5 * n)
    lo, hi = case["arcs_lo"], case["arcs_hi"]
    m = int(case["jobs"] * (hi - lo) / np.log(hi / lo))
    return m // 8, m


def work(case):
    n, m = _size(case)
    b = case.get("offset_bytes", 8) * (n + 1) + 4 * m + 4 * n
    if case.get("weighted") or case["call"] == "f64":
        b += 8 * m
    if case.get("init") == "degree" or case["call"] == "batch":
        b += 4 * n
    if case["call"] == "batch":
        b += 12 * n + 32 * case["graphs"]  # local labels, histogram colours and counts; per-graph words
    return {"bytes": b, "flops": 0}


def _mixer(x, salt):
    """A 64-bit mix of int64 values (wrap-around arithmetic)."""
    x = (x + salt) * -7046029254386353131
    x = x ^ ((x >> 29) & ((1 << 35) - 1))
    x = x * -4658895280553007687
    x = x ^ ((x >> 32) & ((1 << 32) - 1))
    x = x * -7723592293110705685
    return x ^ ((x >> 29) & ((1 << 35) - 1))


def _min_labels(inv, k):
    n = inv.numel()
    first = torch.full((k,), n, dtype=torch.int64, device=inv.device)
    first.scatter_reduce_(0, inv, torch.arange(n, device=inv.device), "amin")
    return first[inv]


def _exact_labels(off, idx, wt=None, init=None, doubles=False):
    """Colour refinement by 64-bit sums: (labels, blocks, rounds)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    off = torch.from_numpy(np.asarray(off).astype(np.int64)).to(dev)
    idx = torch.from_numpy(np.asarray(idx).astype(np.int64)).to(dev)
    n = off.numel() - 1
    if n == 0:
        return np.zeros(0, np.int64), 0, 0
    w = None if wt is None else torch.from_numpy(np.asarray(wt) if doubles else np.asarray(wt).view(np.int64)).to(dev)
    row = torch.repeat_interleave(torch.arange(n, device=dev), off[1:] - off[:-1]) if doubles else None
    col = torch.zeros(n, dtype=torch.int64, device=dev)
    if init is not None:
        col = torch.unique(torch.from_numpy(np.asarray(init).astype(np.int64)).to(dev), return_inverse=True)[1]
    count, rounds = int(col.max()) + 1, 0
    while True:
        salt = 0x1F123BB5 * (rounds + 1)
        if doubles:
            pair, grp = torch.unique(row * count + col[idx], return_inverse=True)
            s = torch.zeros(pair.numel(), dtype=torch.float64, device=dev).index_add_(0, grp, w).float()
            t = _mixer(_mixer(pair % count, salt) ^ s.view(torch.int32).long(), salt + 1)
            sig = torch.zeros(n, dtype=torch.int64, device=dev).index_add_(0, torch.div(pair, count, rounding_mode="floor")[s != 0], t[s != 0])
        else:
            t = _mixer(col[idx], salt)
            t = torch.cumsum(t if w is None else t * w, 0)
            t = torch.cat([torch.zeros(1, dtype=torch.int64, device=dev), t])
            sig = t[off[1:]] - t[off[:-1]]
        vals, inv = torch.unique(_mixer(sig, salt + 2) ^ _mixer(col, salt + 3), return_inverse=True)
        rounds += 1
        new = vals.numel()
        col = inv
        if new == count:
            break
        count = new
    return _min_labels(col, count).cpu().numpy(), count, rounds


def exact(case, seed):
    call = case["call"]
    if call == "edge_batches":
        return None  # the mode's partition is the reference's, not the coarsest one
    if call == "served":
        res = [_exact_labels(off, idx) for off, idx in _mix(case, seed)]
        return dict(labels=[r[0] for r in res], blocks=np.array([r[1] for r in res], dtype=np.int64))
    if call == "batch":
        off, idx, gn, lab = _batch(case, seed)
        labels, blocks, rounds = _exact_labels(off, idx, None, lab)
        n, dev = len(off) - 1, "cuda" if torch.cuda.is_available() else "cpu"
        gn = torch.from_numpy(gn.astype(np.int64)).to(dev)
        g = torch.repeat_interleave(torch.arange(gn.numel() - 1, device=dev), gn[1:] - gn[:-1])
        key, inv, cnt = torch.unique(g * n + torch.from_numpy(labels).to(dev), return_inverse=True, return_counts=True)
        per = torch.bincount(torch.div(key, n, rounding_mode="floor"), minlength=gn.numel() - 1)
        pad = torch.zeros(n - key.numel(), dtype=torch.int64, device=dev)
        res = dict(colors=torch.from_numpy(labels), local=_min_labels(inv, key.numel()) - gn[g], per_graph=per,
                   hist_offsets=torch.cat([per[:1] * 0, torch.cumsum(per, 0)]), hist_colors=torch.cat([key % n, pad]),
                   hist_counts=torch.cat([cnt, pad]))
        return dict({k: v.cpu().numpy() for k, v in res.items()}, fingerprint=None, blocks=blocks, rounds=rounds)
    off, idx = _host_graph(case, seed)
    m = len(idx)
    wt = _doubles(m, seed) if call == "f64" else (_weights(m, seed) if case.get("weighted") else None)
    labels, blocks, rounds = _exact_labels(off, idx, wt, _init(case, off), doubles=call == "f64")
    if call == "noalloc":
        return dict(labels=labels, result=np.array([blocks, rounds, 0, 0]), status=0)
    return dict(labels=labels, blocks=blocks, rounds=rounds)
