"""Delete batches of many vertices around the length that a whole block takes (more than 24 of a vertex), in every
grouping form (8 and 16 thread blocks, and the radix sort past 98,304): heads of long segments at all places of a
thread block's share, segments across two shares, more long segments than blocks. The whole store against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,low,high", [(1, 25, 25), (40, 24, 25), (90, 25, 25), (350, 20, 40), (1500, 25, 25),
                                        (2600, 1, 60), (2600, 25, 37), (4200, 20, 30), (6000, 1, 50)])
def test_long_segments_everywhere(n, low, high):
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    rng = np.random.default_rng(n + high)
    deg = 64
    src = np.repeat(np.arange(n, dtype=np.uint32), deg)
    dst = rng.integers(0, n, len(src)).astype(np.uint32)
    w = np.exp2(rng.uniform(0, 32, len(src))).astype(np.uint64).clip(1, 0xffffffff).astype(np.uint32)
    with Graph(device=0, node2vec=n % 3 == 0) as g:
        ex = po.ExactGraph(n)
        g.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        counts = rng.integers(low, high + 1, n)
        u = np.repeat(np.arange(n, dtype=np.uint32), counts)
        slot = np.concatenate([rng.permutation(deg)[:c] for c in counts]).astype(np.uint32)
        order = rng.permutation(len(u))
        g.delete_batch(u[order], slot[order])
        assert ex.delete(u[order], slot[order]) == 0
        a, b = g.dump(), ex.dump()
        for k in a:
            assert np.array_equal(a[k], b[k]), k
        g.check()
