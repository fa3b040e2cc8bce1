"""The shards of a run are one partition whatever each of them is asked for: some
counted, some delivered as records, on any kernel and with any of the options that
choose one.  (Ranks of one job may differ in them: one prints, the others count.)"""
import pytest

import gmkbe_b200 as G
from gmkbe_b200 import graphgen as gg
from gmkbe_b200.shard import MASK64
from conftest import golden_graph_path

pytestmark = pytest.mark.gpu

MODES = [dict(), dict(collect=True), dict(sharing=False), dict(pair_limit=5000), dict(donate_min_nodes=4)]


def _graph(name):
    if name == "er":
        return gg.erdos_renyi(100, 128, 0.03, 4)
    if name == "wide":
        return gg.erdos_renyi(40, 128, 0.06, 7)
    return gg.read_graph_bin(golden_graph_path(name))


@pytest.mark.parametrize("name", ["er", "wide", "er200", "cl20k_sub"])
@pytest.mark.parametrize("nshards", [2, 5])
def test_shards_of_different_modes_partition_the_set(name, nshards):
    with G.Graph.from_graph(_graph(name)) as g:
        want = g.enumerate(k=1).summary()
        cost = g.root_costs()
        for kw in (dict(), dict(schedule="ordered", task_cost=cost)):
            parts = [[g.enumerate(k=1, shard=s, nshards=nshards, **kw, **m).summary() for m in MODES]
                     for s in range(nshards)]
            for s, p in enumerate(parts):
                assert len(set(p)) == 1, (s, p)      # a shard's own set, in every mode
            c = h = x = 0
            for p in parts:
                c, h, x = c + p[0][0], (h + p[0][1]) & MASK64, x ^ p[0][2]
            assert (c, h, x) == want
