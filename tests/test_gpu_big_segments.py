"""Segments that a whole block appends: long ones (more than 256 edges of one vertex in a batch, at the edges of the
warps' ranges) and single edges that make a large vertex move its store. The whole store against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(g, ex):
    a, b = g.dump(), ex.dump()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def _edges(rng, n, hubs, rest):
    """Batch columns: hubs = {vertex: edges}, rest = edges of random vertices, shuffled together."""
    src = np.concatenate([np.full(c, u, np.uint32) for u, c in hubs.items()] +
                         [rng.integers(0, n, rest).astype(np.uint32)])
    src = src[rng.permutation(len(src))]
    dst = rng.integers(0, n, len(src)).astype(np.uint32)
    w = np.exp2(rng.uniform(0, 32, len(src))).astype(np.uint64).clip(1, 0xffffffff).astype(np.uint32)
    return src, dst, w


@pytest.mark.parametrize("index", [True, False])
@pytest.mark.parametrize("length", [255, 256, 257, 287, 288, 289, 511, 2048, 2049, 9000])
def test_long_segments(length, index):
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    n, rng = 300, np.random.default_rng(length)
    with Graph(device=0, node2vec=index) as g:
        ex = po.ExactGraph(n)
        load = _edges(rng, n, {0: length, 7: 300, 299: 40}, 500)
        g.load_edges(*load, n)
        ex.load(*load)
        _same(g, ex)
        for hubs in ({0: length, 5: length}, {5: 257, 9: 1}):
            ins = _edges(rng, n, hubs, 200)
            assert np.array_equal(g.insert_batch(*ins), ex.insert(*ins))
            _same(g, ex)
        g.check()


@pytest.mark.parametrize("index", [True, False])
def test_large_vertices_move(index):
    """One edge at a time on vertices with thousands of members, through every growth of their arrays, with deletes
    between (lists that shrink and grow back, keys that die in the adjacency index)."""
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    n, rng = 64, np.random.default_rng(4)
    with Graph(device=0, node2vec=index, arena_factor=1.0) as g:
        ex = po.ExactGraph(n)
        load = _edges(rng, n, {u: 1010 + 3 * u for u in range(6)}, 100)
        g.load_edges(*load, n)
        ex.load(*load)
        for step in range(14):
            ins = _edges(rng, n, {u: 1 + step % 3 for u in range(6)}, 5)
            slots = g.insert_batch(*ins)
            assert np.array_equal(slots, ex.insert(*ins))
            if step % 2:
                keep = rng.random(len(slots)) < 0.5
                g.delete_batch(ins[0][keep], slots[keep])
                assert ex.delete(ins[0][keep], slots[keep]) == 0
            _same(g, ex)
        g.check()


def test_many_listed_segments():
    """More listed segments than half the apply kernel's blocks."""
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    n, rng = 1500, np.random.default_rng(6)
    with Graph(device=0, node2vec=False) as g:
        ex = po.ExactGraph(n)
        src = np.repeat(np.arange(n, dtype=np.uint32), 260)
        src = src[rng.permutation(len(src))]
        dst = rng.integers(0, n, len(src)).astype(np.uint32)
        w = rng.integers(1, 1 << 16, len(src)).astype(np.uint32)
        g.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        _same(g, ex)
        ins = _edges(rng, n, {}, 3000)
        assert np.array_equal(g.insert_batch(*ins), ex.insert(*ins))
        _same(g, ex)
