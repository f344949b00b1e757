"""Large copies from and to pageable memory (hostcopy.cu): the same labels as
from page-locked arrays, above and below the size from which threads copy, with
two contexts copying at once."""
import threading

import numpy as np
import pytest

import rbsc_b200 as R

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(a.dtype)
    v[:] = a
    return v


@pytest.mark.parametrize("n,d", [(2000000, 4.9), (2000000, 5.3), (5300000, 2.1)])
def test_pageable_equals_pinned(n, d):
    """Heads of 39 and 42 MB (weights twice that), offsets and labels above and below."""
    off, idx = R.gen_er_host(n, d, seed=n & 7)
    wt = (np.arange(len(idx)) % 5).astype(np.uint64)
    with R.Context(0) as ctx, R.Context(0) as other:
        for w in (wt, None):
            ref = ctx.refine(_pinned(off), _pinned(idx), None if w is None else _pinned(w))
            got, err = [], []

            def call(c):
                try:
                    got.append(c.refine(off, idx, w))
                except Exception as e:  # reported below
                    err.append(e)

            ts = [threading.Thread(target=call, args=(c,)) for c in (ctx, other)]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            assert not err and len(got) == 2
            for r in got:
                assert (r.blocks, r.rounds) == (ref.blocks, ref.rounds) and np.array_equal(r.labels, ref.labels)
