"""How wide the tasks are that a run makes itself.  The thread engine takes a
task's children one after the other and never splits it, so it keeps narrow
ones (16 first-level children) on every schedule; so do runs of the warp engine
that do not share inside a launch: their first launch has no more parallelism than
tasks."""
import pytest

import gmkbe_b200 as G
from gmkbe_b200 import graphgen as gg
from conftest import golden_graph_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["er60", "cl20k_sub"])
def test_thread_engine_tasks_are_sixteen_children_wide(golden, name):
    h = gg.read_graph_bin(golden_graph_path(name))
    nv = h.n - h.n_left
    case = next(c for c in golden["cases"] if c["graph"] == name and c["k"] == 1)
    want = (case["count"], int(case["hash_sum"], 16), int(case["hash_xor"], 16))
    with G.Graph.from_graph(h) as g:
        st = g.enumerate(k=1, engine="thread")
        assert st.summary() == want
        per_root = -(-8 * st.threads // h.n_left)
        width = max(16, -(-nv // per_root))
        assert st.tasks == h.n_left * -(-nv // width)
        # planned: the roots that cost more than a share are cut as narrow as that
        st = g.enumerate(k=1, engine="thread", schedule="ordered", task_cost=g.root_costs(),
                         tasks_per_worker=1 << 20)
        assert st.summary() == want
        m = max(1, nv // 16)
        assert st.tasks == h.n_left * -(-nv // -(-nv // m))


@pytest.mark.parametrize("kw", [dict(collect=True), dict(sharing=False)])
def test_tasks_of_runs_without_sharing_are_sixteen_children_wide(kw):
    g = gg.erdos_renyi(60, 150, 0.02, 5)
    nv = g.n - g.n_left
    with G.Graph.from_graph(g) as dg:
        want = dg.enumerate(k=1).summary()
        # (nothing is split, so the tasks are the first launch's)
        st = dg.enumerate(k=1, split_min_nodes=0xFFFFFFFF, **kw)
        assert st.summary() == want and st.rounds == 1
        assert st.tasks == g.n_left * -(-nv // 16)
        st = dg.enumerate(k=1, split_min_nodes=0xFFFFFFFF, schedule="ordered", task_cost=dg.root_costs(),
                          tasks_per_worker=1 << 20, **kw)
        assert st.summary() == want and st.rounds == 1
        assert st.tasks == g.n_left * -(-nv // -(-nv // (nv // 16)))
