"""A result limit on a small graph whose tasks are short (a few search nodes each):
the run ends soon after its results are found, not when the whole graph has been
searched, and a capped graph of a batch ends alone."""
import numpy as np
import pytest

import gmkbe_b200 as G
from gmkbe_b200 import graphgen as gg

pytestmark = pytest.mark.gpu


def _sparse(n, m):
    rng = np.random.default_rng(n)
    return gg.relabel(np.concatenate([np.arange(n), rng.integers(0, n, m - n)]),
                      np.concatenate([np.arange(n), rng.integers(0, n, m - n)]))


@pytest.mark.parametrize("kw", [dict(), dict(chunk=1)])
def test_a_limit_ends_a_run_of_short_tasks(kw):
    with G.Graph.from_graph(_sparse(128, 300)) as g:
        full = g.enumerate(k=1, threads=64 * 32, **kw)
        assert not full.truncated
        for limit in (1, 64, 1000):
            # 64 warps: a few results and a few nodes each beyond the limit
            st = g.enumerate(k=1, threads=64 * 32, result_limit=limit, **kw)
            assert st.count == limit and st.truncated
            assert st.nodes < full.nodes // 2
        st = g.enumerate(k=1, result_limit=1, **kw)
        assert st.count == 1 and st.truncated and st.nodes < full.nodes


def test_a_capped_graph_of_a_batch_ends_alone():
    with G.Graph.from_graph(_sparse(128, 300)) as a, G.Graph.from_graph(_sparse(120, 290)) as b:
        fa, fb = G.enumerate_batch([a, b], [1, 1])
        ca, cb = G.enumerate_batch([a, b], [1, 1], limits=[1, 0], threads=64 * 32)
        assert ca.count == 1 and ca.truncated and ca.nodes < fa.nodes // 2
        assert cb.summary() == fb.summary() and cb.nodes == fb.nodes
