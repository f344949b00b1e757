"""A context frees its graphs when it closes (an error inside a `with` leaves
them behind), and they answer with an error from then on."""
import subprocess
import sys

import pytest

import rbsc_b200 as R
from rbsc_b200 import graphs as G

pytestmark = pytest.mark.gpu

# (in a process of its own: a graph freed after its context can end the process)
LEFT_BEHIND = """
import gc
import rbsc_b200 as R
from rbsc_b200 import graphs as G
for _ in range(20):
    try:
        with R.Context(0) as ctx:
            kept = [ctx.upload(*G.er_directed(n, 4 * n, seed=n)) for n in (500, 30000, 200000)]
            for g in kept:
                g.refine()
            raise ValueError
    except ValueError:
        pass
    kept = g = None
    gc.collect()
print("done")
"""


def test_graphs_left_behind():
    r = subprocess.run([sys.executable, "-c", LEFT_BEHIND], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "done\n", r.stderr


def test_a_closed_graph_answers_with_an_error():
    off, idx = G.er_directed(500, 2000, seed=1)
    with R.Context(0) as ctx:
        g = ctx.upload(off, idx)
        want = g.refine().blocks
    for call in (g.refine, g.refine_device):
        with pytest.raises(R.RbscError):
            call()
    g.free()
    with R.Context(0) as ctx:
        assert ctx.refine(off, idx).blocks == want
