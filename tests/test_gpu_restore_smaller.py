"""A handle with a minimum arena size that held a large graph restores a small one: the arenas grow to the minimum with
nothing in them (the large graph's extent is not copied)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [True, False])
@pytest.mark.parametrize("arena_mb", [16, 48, 400])
def test_restore_small_over_large(arena_mb, index, tmp_path):
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    rng = np.random.default_rng(5)
    n, m = 500, 4000
    small = (rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32),
             rng.integers(1, 1 << 20, m).astype(np.uint32))
    path = str(tmp_path / "small.bin")
    with Graph(device=0, node2vec=index) as g:
        g.load_edges(*small, n)
        g.save(path)
    ex = po.ExactGraph(n)
    ex.load(*small)
    bn, bm = 5000, 3_000_000
    big = (rng.integers(0, bn, bm).astype(np.uint32), rng.integers(0, bn, bm).astype(np.uint32),
           rng.integers(1, 1 << 20, bm).astype(np.uint32))
    with Graph(device=0, node2vec=index, arena_bytes=arena_mb << 20) as g:
        for _ in range(2):
            g.load_edges(*big, bn)
            g.restore(path)
            assert g.stats()["arena_bytes"] >= (arena_mb << 20) * 0.99
            g.check()
            batch = tuple(x[:900] % n + 1 if i == 2 else x[:900] % n for i, x in enumerate(big))
            e2 = po.ExactGraph(n)
            e2.load(*small)
            assert np.array_equal(g.insert_batch(*batch), e2.insert(*batch))
            a, b = g.dump(), e2.dump()
            for k in a:
                assert np.array_equal(a[k], b[k]), k
