"""The adjacency index under steady turnover: the same edges inserted and deleted again and again rebuild a vertex's
table in place (its live keys always fit), so the store stops growing; walks and the whole store stay the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 3, 4, 7, 8, 15, 16, 31, 400])
def test_turnover_rebuilds_in_place(degree):
    from bingo_b200 import NODE2VEC, Graph
    from oracle import pyoracle as po
    n, rng = 40, np.random.default_rng(degree)
    with Graph(device=0, node2vec=True) as g:
        ex = po.ExactGraph(n)
        src = np.repeat(np.arange(n, dtype=np.uint32), degree)
        dst = rng.integers(0, n, len(src)).astype(np.uint32)
        w = rng.integers(1, 9, len(src)).astype(np.uint32)
        g.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        u = np.repeat(np.arange(n, dtype=np.uint32), 2)
        used = []
        for turn in range(12):
            v = ((u * 7 + np.arange(len(u)) + 3 * (turn % 4)) % n).astype(np.uint32)  # new keys for four turns
            ww = np.full(len(u), 4, np.uint32)
            slots = g.insert_batch(u, v, ww)
            assert np.array_equal(slots, ex.insert(u, v, ww))
            g.delete_batch(u, slots)
            assert ex.delete(u, slots) == 0
            g.check()
            used.append(g.stats()["arena_used"])
        a, b = g.dump(), ex.dump()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
        starts = np.arange(n, dtype=np.uint32)
        assert np.array_equal(g.walk(app=NODE2VEC, length=20, starts=starts, seed=1, p=0.5, q=2.0),
                              ex.walk(1, 20, starts, seed=1, p=0.5, q=2.0))
        slots_left = 24 * 16 + 24 * 4  # slot and back-pointer growth of a vertex over the turns, at most doubled
        assert used[-1] - used[3] <= n * 4 * slots_left
