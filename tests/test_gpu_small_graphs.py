"""The bit-mask search of small graphs (at most 128 vertices a side, count mode):
sides at the edges of its mask words, every form of task and limit it takes,
against the oracle and against the list-based search (which a run without
in-launch sharing keeps)."""
import numpy as np
import pytest

import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg
from gmkbe_b200.shard import MASK64

pytestmark = pytest.mark.gpu


def _sparse(nu, nv, seed):
    """Every vertex keeps an edge, so both sides have exactly nu and nv vertices:
    a path-like cover plus a few random edges (few results at k = 1)."""
    rng = np.random.default_rng(seed)
    m = max(nu, nv)
    u, v = np.arange(m) % nu, np.arange(m) % nv
    extra = m // 8
    return gg.relabel(np.concatenate([u, rng.integers(0, nu, extra)]),
                      np.concatenate([v, rng.integers(0, nv, extra)]))


SIDES = [(1, 1), (1, 32), (32, 1), (31, 33), (32, 32), (33, 31), (64, 20), (20, 64), (65, 33), (64, 64),
         (127, 40), (40, 128), (129, 40), (40, 129)]


@pytest.mark.parametrize("nu,nv", SIDES)
def test_sides_at_the_mask_word_edges(nu, nv):
    g = _sparse(nu, nv, 7 * nu + nv)
    assert (g.n_left, g.n - g.n_left) == (nu, nv)
    want = O.enumerate_oracle(g, 1).summary()
    with G.Graph.from_graph(g) as dg:
        assert dg.enumerate(k=1).summary() == want
        assert dg.enumerate(k=1, schedule="plain").summary() == want
        assert dg.enumerate(k=1, sharing=False).summary() == want


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("nu,nv,p", [(9, 12, 0.4), (12, 9, 0.25), (14, 11, 0.7)])
def test_every_k_against_the_oracle(nu, nv, p, k):
    g = gg.erdos_renyi(nu, nv, p, 40 + k)
    want = O.enumerate_oracle(g, k).summary()
    with G.Graph.from_graph(g) as dg:
        assert dg.enumerate(k=k).summary() == want
        assert dg.enumerate(k=k, sharing=False).summary() == want


def test_complete_and_star_graphs():
    u, v = np.meshgrid(np.arange(40), np.arange(70), indexing="ij")
    with G.Graph.from_graph(gg.relabel(u.ravel(), v.ravel())) as dg:
        for k in (1, 5, 15):
            assert dg.enumerate(k=k).count == 1
    star = gg.relabel(np.zeros(100, np.int64), np.arange(100))
    with G.Graph.from_graph(star) as dg:
        assert dg.enumerate(k=1).summary() == O.enumerate_oracle(star, 1).summary()


@pytest.mark.parametrize("nu,nv,k", [(28, 30, 2), (40, 50, 1), (80, 100, 1)])
def test_forms_of_tasks_agree(nu, nv, k):
    g = gg.erdos_renyi(nu, nv, 3.0 / nv, 5)
    with G.Graph.from_graph(g) as dg:
        ref = dg.enumerate(k=k, sharing=False)
        want = ref.summary()
        cost = dg.root_costs()
        log = np.zeros(g.n_left, np.uint64)
        st = dg.enumerate(k=k, root_nodes=log)
        assert st.summary() == want and log.sum() == st.nodes and (log > 0).all()
        for kw in (dict(chunk=1), dict(chunk=7), dict(threads=32), dict(threads=4096),
                   dict(schedule="ordered", task_cost=cost), dict(schedule="plain", task_cost=cost),
                   dict(donate_min_nodes=64), dict(tasks_per_worker=1)):
            assert dg.enumerate(k=k, **kw).summary() == want, kw
        mid = g.n_left // 3
        parts = [dg.enumerate(k=k, root_begin=0, root_end=mid), dg.enumerate(k=k, root_begin=mid)]
        parts2 = [dg.enumerate(k=k, shard=s, nshards=3) for s in range(3)]
        tasks = G.plan_tasks(g.n, g.n_left, cost, target_tasks=300)
        parts3 = [dg.enumerate(k=k, tasks=tasks[i::2]) for i in range(2)]
        for ps in (parts, parts2, parts3):
            xor = 0
            for p in ps:
                xor ^= p.hash_xor
            assert (sum(p.count for p in ps), sum(p.hash_sum for p in ps) & MASK64, xor) == want
        for limit in (1, 100, want[0] // 2, want[0], want[0] + 1):
            st = dg.enumerate(k=k, result_limit=limit)
            assert st.count == min(limit, want[0]) and st.truncated == (limit <= want[0])
        assert dg.enumerate(k=k).summary() == want


def test_deep_stacks_reach_the_spill_area():
    # nearly complete graphs: each included vertex leaves a state behind, more
    # of them than the stack's shared part holds
    u, v = np.meshgrid(np.arange(30), np.arange(34), indexing="ij")
    keep = (u.ravel() + v.ravel()) % 17 != 0
    keep &= ~((u.ravel() < 6) & (v.ravel() < 6))
    g = gg.relabel(u.ravel()[keep], v.ravel()[keep])
    for k in (1, 2):
        with G.Graph.from_graph(g) as dg:
            a = dg.enumerate(k=k, schedule="plain", result_limit=300_000, watchdog_ms=20_000)
            b = dg.enumerate(k=k, sharing=False, result_limit=300_000, watchdog_ms=20_000)
            assert a.count == b.count and a.truncated == b.truncated
            if not a.truncated:
                assert a.summary() == b.summary()


def test_batches_of_small_graphs_and_mixed_sizes():
    gs = [gg.erdos_renyi(n, n + 3, 2.5 / n, n) for n in (6, 20, 31, 33, 50, 70)]
    ks = [3, 2, 1, 2, 1, 1]
    dgs = [G.Graph.from_graph(g) for g in gs]
    try:
        want = [dg.enumerate(k=k, sharing=False).summary() for dg, k in zip(dgs, ks)]
        for n in (4, 6):      # up to 36 vertices a side, up to 73
            got = G.enumerate_batch(dgs[:n], ks[:n])
            assert [st.summary() for st in got] == want[:n]
        caps = [max(1, w[0] // 2) if i % 2 else w[0] + 1 for i, w in enumerate(want)]
        for w, cap, st in zip(want, caps, G.enumerate_batch(dgs, ks, limits=caps)):
            assert st.count == min(w[0], cap) and st.truncated == (cap <= w[0])
            if cap > w[0]:
                assert st.summary() == w
    finally:
        for dg in dgs:
            dg.close()


@pytest.mark.parametrize("nu,nv,m,k", [(32, 33, 60, 2), (33, 32, 150, 1), (64, 65, 200, 1), (40, 33, 70, 2),
                                       (34, 12, 60, 3), (96, 97, 330, 1), (128, 127, 400, 1), (65, 20, 90, 2)])
def test_fans_of_children(nu, nv, m, k):
    # sparse sides over a mask word: an included vertex misses many candidates,
    # of which one at most can join; whole, shared early, in parts and cut off
    rng = np.random.default_rng(nu * nv + k)
    u = np.concatenate([np.arange(nu), rng.integers(0, nu, m - nu)])
    v = np.concatenate([np.arange(nu) % nv, rng.integers(0, nv, m - nu)])
    g = gg.relabel(u, v)
    with G.Graph.from_graph(g) as dg:
        want = dg.enumerate(k=k, sharing=False).summary()
        for kw in (dict(), dict(donate_min_nodes=64), dict(chunk=3), dict(threads=32), dict(schedule="plain")):
            assert dg.enumerate(k=k, **kw).summary() == want, kw
        st = dg.enumerate(k=k, result_limit=want[0] // 2)
        assert st.count == want[0] // 2 and st.truncated
        with G.Graph.from_graph(g) as other:
            assert [s.summary() for s in G.enumerate_batch([dg, other], [k, k])] == [want, want]
