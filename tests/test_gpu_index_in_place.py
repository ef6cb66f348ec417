"""The adjacency index of vertices whose edges come and go: each turn inserts edges to ids never seen before and
deletes them again, so that dead keys fill the tables while the live keys fit. The tables are rebuilt where they are:
the index arena (a handle with the index against one without, same calls) does not grow past the first turns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (degree, edges added per turn and vertex, vertices): by one warp, and the last three by a whole block (long tables).
@pytest.mark.parametrize("degree,add,hubs", [(1, 1, 40), (2, 2, 40), (3, 2, 40), (6, 2, 40), (7, 1, 40), (13, 3, 40),
                                             (30, 2, 40), (100, 28, 9), (700, 200, 5), (3000, 750, 3), (7000, 300, 2)])
def test_index_does_not_grow(degree, add, hubs):
    from bingo_b200 import NODE2VEC, Graph
    from oracle import pyoracle as po
    n, rng = 200_000, np.random.default_rng(degree)
    src = np.repeat(np.arange(hubs, dtype=np.uint32), degree)
    dst = np.concatenate([rng.permutation(hubs + degree)[:degree] for _ in range(hubs)]).astype(np.uint32)
    w = rng.integers(1, 9, len(src)).astype(np.uint32)
    u = np.repeat(np.arange(hubs, dtype=np.uint32), add)
    ww = np.full(len(u), 4, np.uint32)
    with Graph(device=0, node2vec=True) as g, Graph(device=0, node2vec=False) as plain:
        ex = po.ExactGraph(n)
        for x in (g, plain):
            x.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        cap = 1 << (2 * (degree + add) - 1).bit_length()
        turns = 4 + 3 * (cap // 2 // add + 1)  # the new keys would fill half the table three times
        fresh, used = 10_000, []
        for turn in range(turns):
            v = (fresh + np.arange(len(u))).astype(np.uint32) % n
            fresh = 10_000 if fresh + 2 * len(u) > n else fresh + len(u)
            slots = g.insert_batch(u, v, ww)
            assert np.array_equal(slots, plain.insert_batch(u, v, ww))
            assert np.array_equal(slots, ex.insert(u, v, ww))
            for x in (g, plain):
                x.delete_batch(u, slots)
            assert ex.delete(u, slots) == 0
            used.append(g.stats()["arena_used"] - plain.stats()["arena_used"])
        g.check()
        a, b = g.dump(), ex.dump()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
        starts = np.arange(hubs, dtype=np.uint32)
        assert np.array_equal(g.walk(app=NODE2VEC, length=20, starts=starts, seed=1, p=0.5, q=2.0),
                              ex.walk(1, 20, starts, seed=1, p=0.5, q=2.0))
        assert used[-1] == used[3]
