"""The thread engine at every k that it takes, against the oracle: k + 1 sources of
outside vertices, more than four of them from k = 4 on.  The same search runs in the
call that allocates nothing."""
import pytest

import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv,p,k", [(6, 14, 0.5, 4), (9, 8, 0.8, 4), (8, 9, 0.85, 5), (9, 9, 0.9, 6), (10, 10, 0.95, 7),
                                       (11, 11, 1.0, 8)])
def test_thread_engine_past_four_sources(nu, nv, p, k):
    g = gg.erdos_renyi(nu, nv, p, 3)
    with G.Graph.from_graph(g) as dg:
        assert dg.enumerate(k=k, engine="thread").summary() == O.enumerate_oracle(g, k).summary()
