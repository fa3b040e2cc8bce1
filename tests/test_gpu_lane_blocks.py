"""Children of a global side decided 32 at a time, one per lane, and the bit-mask
search of nodes with at most 32 vertices a side (list-based kernel): graphs at
the edges of their limits, in count and record mode, with split and shared
trees, against the oracle.  arena_words keeps small graphs on that kernel."""
import numpy as np
import pytest

import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg

pytestmark = pytest.mark.gpu

LIST = dict(arena_words=1 << 18)


def _check(g, k, records=True):
    want = O.enumerate_oracle(g, k).summary()
    with G.Graph.from_graph(g) as dg:
        for kw in (dict(), dict(chunk=1), dict(chunk=33), dict(donate_min_nodes=1),
                   dict(sharing=False, split_min_nodes=1), dict(sharing=False, split_min_nodes=3, chunk=2),
                   dict(schedule="plain"), dict(threads=64)):
            assert dg.enumerate(k=k, **LIST, **kw).summary() == want, kw
        if not records:
            return
        for kw in (dict(), dict(out_words=160, threads=64), dict(schedule="plain")):
            sets = []
            st = dg.enumerate(k=k, sink=lambda x, y: sets.append((x, y)) and False, **LIST, **kw)
            assert st.summary() == want, kw
            assert len(sets) == want[0] and O.set_summary(sets) == want, kw
        st = dg.enumerate(k=k, result_limit=max(1, want[0] // 2), collect=True, **LIST)
        assert st.count == len(st.results) == len(set(st.results)) == max(1, want[0] // 2)


@pytest.mark.parametrize("nu,nv,deg,k,seed", [
    (40, 45, 2.0, 1, 1), (30, 70, 3.0, 1, 2), (70, 30, 3.0, 1, 3), (35, 35, 6.0, 1, 4), (16, 18, 2.0, 2, 5),
    (14, 14, 4.0, 2, 6), (10, 12, 2.5, 3, 7), (9, 8, 4.0, 3, 8), (7, 7, 2.5, 4, 9)])
def test_random_graphs(nu, nv, deg, k, seed):
    _check(gg.erdos_renyi(nu, nv, deg / nv, seed), k, records=O.enumerate_oracle(
        gg.erdos_renyi(nu, nv, deg / nv, seed), k).count < 30_000)


@pytest.mark.parametrize("k", [1, 2])
def test_power_law_graphs(k):
    nu, nv, m = (90, 140, 230) if k == 1 else (24, 30, 48)
    _check(gg.chung_lu(nu, nv, m, 2.1, 17, max_deg=40), k, records=k == 1)


@pytest.mark.parametrize("d", [31, 32, 33, 63, 64, 65, 66])
def test_rows_and_lists_at_their_limits(d):
    # a V hub with d neighbours beside a U vertex with d neighbours and a sparse
    # rest: rows of d entries are walked by one lane (32), filtered into a list of
    # at most 64, or make a universe of 32 vertices too large
    u = np.concatenate([np.arange(d), np.full(d, d), np.arange(d + 1, d + 6)])
    v = np.concatenate([np.zeros(d, np.int64), 1 + np.arange(d), 1 + np.arange(5)])
    _check(gg.relabel(u, v), 1, records=False)


@pytest.mark.parametrize("k", [8, 9, 10, 15])
def test_large_k(k):
    # miss counts are kept in four bits up to k = 9; larger ones are built child
    # by child
    _check(gg.erdos_renyi(11, 10, 0.5, k), k)
    _check(gg.erdos_renyi(12, 3, 0.4, k), k)


@pytest.mark.parametrize("nu,nv,p", [(8, 70, 0.5), (70, 8, 0.5), (10, 60, 0.4)])
def test_many_outsiders(nu, nv, p):
    # a few vertices against many: most of the long side are outsiders of most
    # nodes, more than the 32 a warp's lanes hold
    _check(gg.erdos_renyi(nu, nv, p, 4), 1, records=False)


def test_larger_than_the_small_graph_search():
    # 129 vertices a side and more: the same kernel without being asked for
    for g in (gg.relabel(np.arange(130), np.arange(130)), gg.erdos_renyi(140, 135, 1.5 / 135, 5),
              gg.chung_lu(150, 260, 420, 2.1, 31, max_deg=30)):
        want = O.enumerate_oracle(g, 1).summary()
        with G.Graph.from_graph(g) as dg:
            cost = dg.root_costs()
            log = np.zeros(g.n_left, np.uint64)
            st = dg.enumerate(k=1, root_nodes=log)
            assert st.summary() == want and log.sum() == st.nodes and (log > 0).all()
            assert dg.enumerate(k=1, chunk=17).nodes == dg.enumerate(k=1, chunk=17, donate_min_nodes=1).nodes
            assert dg.enumerate(k=1, schedule="ordered", task_cost=cost).summary() == want
            got = G.enumerate_batch([dg], [1])[0]
            assert got.summary() == want


def test_a_reached_limit_ends_long_rows():
    # three V hubs adjacent to 20 000 U vertices: lists of that length are being
    # built when the limit is reached, and those tasks are dropped; the run, and
    # in a batch the graph, stops at its cap while the other graph runs to its end
    hub = gg.hubs_and_sparse(3, 40, 20_000, 3, 6)
    small = gg.erdos_renyi(12, 140, 2.0 / 140, 9)
    want = O.enumerate_oracle(small, 1).summary()
    with G.Graph.from_graph(hub) as h, G.Graph.from_graph(small) as s:
        for limit in (1, 1000, 200_000):
            st = h.enumerate(k=2, result_limit=limit)
            assert st.count == limit and st.truncated
        got = G.enumerate_batch([h, s], [2, 1], limits=[5000, 0])
        assert got[0].count == 5000 and got[0].truncated
        assert got[1].summary() == want and not got[1].truncated
        assert h.enumerate(k=2, result_limit=50, collect=True).count == 50
