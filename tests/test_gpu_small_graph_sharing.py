"""Sharing of search states between the warps of the small graphs' search: runs
that make its workspace grow (in a process of their own, so that the workspace
starts empty), and runs that hand on more states than there are slots for."""
import os
import subprocess
import sys

import pytest

import gmkbe_b200 as G
from gmkbe_b200 import graphgen as gg
from conftest import ROOT

pytestmark = pytest.mark.gpu

GROW = """
import numpy as np
import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg

def graph(nu, nv, m, seed):
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.arange(nu), rng.integers(0, nu, m - nu)])
    v = np.concatenate([np.arange(nu) % nv, rng.integers(0, nv, m - nu)])
    return gg.relabel(u, v)

# a few warps, then the whole GPU; wide masks (few warps per SM), then narrow ones (many)
runs = [(graph(30, 28, 60, 1), 1, 32), (graph(30, 28, 60, 1), 1, 0), (graph(100, 120, 150, 2), 1, 0),
        (graph(20, 18, 40, 3), 2, 0), (graph(50, 60, 80, 4), 1, 1024), (graph(50, 60, 80, 4), 1, 0),
        (graph(20, 18, 40, 3), 2, 0)]
want = [O.enumerate_oracle(g, k).summary() for g, k, _ in runs]
for (g, k, threads), w in zip(runs, want):
    with G.Graph.from_graph(g) as dg:
        for _ in range(5):
            assert dg.enumerate(k=k, threads=threads).summary() == w, (g.n, k, threads)
print("ok")
"""


def test_runs_that_grow_the_workspace():
    out = subprocess.run([sys.executable, "-c", GROW], capture_output=True, text=True, cwd=ROOT,
                         env=dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.path.join(ROOT, "tests")),
                         timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]


@pytest.mark.parametrize("nu,nv,p", [(80, 80, 0.35), (64, 60, 0.5)])
def test_states_handed_on_past_the_last_slot(nu, nv, p):
    # 64 slots a warp, rounded up to a power of two: the tickets go past the last
    # slot, and the next launch starts from the marks that this one left
    with G.Graph.from_graph(gg.erdos_renyi(nu, nv, p, 3)) as dg:
        want = dg.enumerate(k=1, sharing=False).summary()
        for _ in range(2):
            st = dg.enumerate(k=1, watchdog_ms=60_000)
            assert st.summary() == want
            assert st.donations > 1 << (64 * (st.threads // 32) - 1).bit_length()
