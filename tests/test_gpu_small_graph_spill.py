"""The part of the small graphs' search stack that lies past shared memory: graphs
whose search is deeper than it, enumerated completely, against the oracle or the
list-based search.  How deep the search goes is found by restating its steps here."""
import numpy as np
import pytest

import gmkbe_b200 as G
import oracle as O
from gmkbe_b200 import graphgen as gg

pytestmark = pytest.mark.gpu

SHARED = {1: 64, 2: 32, 3: 16, 4: 16}     # stack entries in shared memory, by mask words a side


def _missing_stars(pieces, extra):
    """U: one vertex f next to all of V and one centre a piece; V: `pieces[i]` vertices
    that centre i misses (and no other does), and `extra` next to f alone.  At k = 1 a
    result takes a centre and one of its piece, or the whole piece without the centre."""
    edges = [(0, v) for v in range(sum(pieces) + extra)]
    first = 0
    for i, n in enumerate(pieces):
        edges += [(1 + i, v) for v in range(sum(pieces)) if not first <= v < first + n]
        first += n
    e = np.array(edges)
    return gg.relabel(e[:, 0], e[:, 1])


def _bits(m):
    while m:
        yield (m & -m).bit_length() - 1
        m &= m - 1


def _depth(g, k, root, max_nodes):
    """(entries on the stack at most, fans among them) over the first `max_nodes` nodes
    of the search of one root (the steps of enum_dense.cuh for two or more words)."""
    nl, nv = g.n_left, g.n - g.n_left
    miss = [[(1 << nv) - 1] * nl, [(1 << nl) - 1] * nv]
    for u in range(nl):
        for y in g.adj[g.offsets[u]:g.offsets[u + 1]]:
            miss[0][u] &= ~(1 << (int(y) - nl))
            miss[1][int(y) - nl] &= ~(1 << u)
    size = (nl, nv)

    def refit(inc, can):
        full = [sum(1 << v for v in _bits(inc[s]) if (miss[s][v] & inc[1 - s]).bit_count() >= k) for s in (0, 1)]
        return [sum(1 << v for v in _bits(can[s]) if (miss[s][v] & inc[1 - s]).bit_count() <= k
                    and not miss[s][v] & full[1 - s]) for s in (0, 1)]

    state = ([1 << root, 0], [(1 << nl) - (2 << root), (1 << nv) - 1])
    stack, deep, fans = [], 0, 0
    for _ in range(max_nodes):
        if state is None:
            if not stack:
                break
            inc, can, side, left = stack[-1]
            if left:
                v = left & -left
                stack[-1][3] = left & (left - 1)
                state = ([inc[s] | (v if s == side else 0) for s in (0, 1)], can)
            else:
                state = (inc, can)
                stack.pop()
        inc, can = list(state[0]), refit(*state)
        state = None
        all_ = [inc[s] | can[s] for s in (0, 1)]
        if not all_[1]:
            continue
        t = [[(miss[s][v] & all_[1 - s]).bit_count() for v in range(size[s])] for s in (0, 1)]
        hard = [sum(1 << v for v in _bits(all_[s]) if t[s][v] >= k) for s in (0, 1)]
        bad = [sum(1 << v for v in _bits(all_[s]) if t[s][v] > k) for s in (0, 1)]
        if any(t[s][v] <= k and not miss[s][v] & hard[1 - s]
               for s in (0, 1) for v in range(size[s]) if not all_[s] >> v & 1):
            continue
        if not (bad[0] | bad[1]):
            continue
        for s in (0, 1):
            forced = sum(1 << v for v in _bits(can[s]) if t[s][v] <= k and not miss[s][v] & bad[1 - s])
            inc[s] |= forced
            can[s] &= ~forced
        if can[0].bit_count() + can[1].bit_count() <= 5:
            continue
        worst = max(((t[s][v], -s, -v) for s in (0, 1) for v in _bits(inc[s] & bad[s])), default=None)
        pick = list(can)
        if worst:
            s, v = -worst[1], -worst[2]
            pick = [0, 0]
            pick[1 - s] = can[1 - s] & miss[s][v]
            if (miss[s][v] & inc[1 - s]).bit_count() + 1 == k and pick[1 - s].bit_count() >= 6:
                can = [can[x] & ~pick[x] for x in (0, 1)]
                stack.append([inc, can, 1 - s, pick[1 - s]])
                deep = max(deep, len(stack))
                fans = max(fans, sum(1 for e in stack[SHARED[3]:] if e[3]))
                continue
        _, s, v = max((t[s][v], -s, -v) for s in (0, 1) for v in _bits(pick[s]))
        s, v = -s, -v
        can[s] &= ~(1 << v)
        stack.append([list(inc), list(can), 0, 0])
        deep = max(deep, len(stack))
        inc[s] |= 1 << v
        state = (inc, can)
    return deep, fans


CASES = {"pairs_3_words": ([2] * 12, 45), "pairs_4_words": ([2] * 12, 75), "fans": ([6] * 9, 12)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_search_past_the_shared_part_of_the_stack(name):
    g = _missing_stars(*CASES[name])
    words = (max(g.n_left, g.n - g.n_left) + 31) // 32
    assert words in (3, 4)
    depth, fans = max(_depth(g, 1, r, 300) for r in range(3))
    assert depth > SHARED[words] and (fans > 0) == (name == "fans")
    with G.Graph.from_graph(g) as dg:
        want = dg.enumerate(k=1, sharing=False, watchdog_ms=60_000).summary()
        if name != "fans":
            assert want == O.enumerate_oracle(g, 1).summary()
        for kw in (dict(), dict(threads=256 * 32), dict(donate_min_nodes=64), dict(chunk=1000),
                   *([] if name == "fans" else [dict(schedule="plain"), dict(threads=8 * 32)])):
            assert dg.enumerate(k=1, watchdog_ms=60_000, **kw).summary() == want, kw
