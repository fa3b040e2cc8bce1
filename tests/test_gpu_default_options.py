"""An option given its documented default is the same run as without it, on the
small graphs' kernel too, and the autotuner's defaults are that run."""
import numpy as np
import pytest

import gmkbe_b200 as G
from gmkbe_b200 import autotune
from gmkbe_b200 import graphgen as gg
from conftest import golden_graph_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,k", [("southernwomen", 1), ("er60", 2), ("crime", 1)])
def test_defaults_given_or_not_are_one_run(name, k):
    h = gg.read_graph_bin(golden_graph_path(name))
    with G.Graph.from_graph(h) as g:
        # (the node count tells the kernels apart, and depends on nothing else here)
        def run(**kw):
            st = g.enumerate(k=k, **kw)
            return st.summary(), st.nodes, st.threads
        want = run()
        for kw in (dict(pair_limit=4096), dict(bits_min_list=64), dict(pair_limit=4096, bits_min_list=64),
                   dict(tasks_per_worker=8), dict(split_min_nodes=64)):
            assert run(**kw) == want, kw
        cost = g.root_costs()
        tuned = autotune.apply(g, autotune.DEFAULTS, cost, autotune.degree_buckets(h, h.n_left), want[2])
        assert run(**tuned) == run(schedule="ordered", task_cost=cost)
        # another value is the list-based search's rule, and the same set
        other = run(pair_limit=4095)
        assert other[0] == want[0]
        if max(h.n_left, h.n - h.n_left) <= 128:
            assert other[1:] != want[1:]
