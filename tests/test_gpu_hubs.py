"""Hubs with more than 128 leaves: frames whose children nothing bounds, so they are
built one by one -- shared, split between launches, in small arenas and as records,
against the oracle; and more members than a lane block takes (15)."""
import numpy as np
import pytest

import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg

pytestmark = pytest.mark.gpu


def _star(leaves, flip):
    a, b = np.zeros(leaves, np.int64), np.arange(leaves)
    return gg.relabel(b, a) if flip else gg.relabel(a, b)


GRAPHS = {
    "star_v": (lambda: _star(140, False), 1),
    "star_u": (lambda: _star(140, True), 1),
    "star_k2": (lambda: _star(135, False), 2),
    "two_hubs": (lambda: gg.hubs_and_sparse(2, 70, 140, 2, 3), 1),
    "three_hubs": (lambda: gg.hubs_and_sparse(3, 31, 145, 2, 7), 1),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_hubs_against_the_oracle(name):
    make, k = GRAPHS[name]
    h = make()
    assert max(h.n_left, h.n - h.n_left) > 128
    want = O.enumerate_oracle(h, k).summary()
    with G.Graph.from_graph(h) as g:
        for kw in (dict(), dict(donate_min_nodes=1), dict(threads=64 * 32), dict(sharing=False, split_min_nodes=4),
                   dict(chunk=1), dict(chunk=1000), dict(schedule="ordered", task_cost=g.root_costs())):
            assert g.enumerate(k=k, watchdog_ms=60_000, **kw).summary() == want, kw
        for words in (1024, 2048):
            assert g.enumerate(k=k, arena_words=words, watchdog_ms=60_000).summary() == want
        st = g.enumerate(k=k, collect=True, watchdog_ms=60_000)
        assert O.set_summary(st.results) == want
