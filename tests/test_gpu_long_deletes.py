"""Deletes of one vertex by one warp (up to 24 in a batch) and by a whole block (more): at the line between them, at
chunks of 32, with absent, repeated and already deleted slots mixed in, lists emptied to the last member. The whole
store against the oracle after every batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(g, ex):
    a, b = g.dump(), ex.dump()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("index", [True, False])
@pytest.mark.parametrize("count", [1, 2, 23, 24, 25, 31, 32, 33, 64, 65, 400, 999])
def test_deletes_of_hubs(count, index):
    from bingo_b200 import BingoError, Graph
    from oracle import pyoracle as po
    n, rng = 50, np.random.default_rng(count)
    deg = 1000
    src = np.concatenate([np.full(deg, u, np.uint32) for u in (0, 3, 49)] + [rng.integers(0, n, 300).astype(np.uint32)])
    src = src[rng.permutation(len(src))]
    dst = rng.integers(0, n, len(src)).astype(np.uint32)
    w = np.where(rng.random(len(src)) < 0.5, rng.integers(1, 8, len(src)),
                 np.exp2(rng.uniform(0, 32, len(src))).astype(np.uint64).clip(1, 0xffffffff)).astype(np.uint32)
    with Graph(device=0, node2vec=index) as g:
        ex = po.ExactGraph(n)
        g.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        for turn in range(3):
            # Hub slots anywhere, at the front and at the end, some repeated, some absent; others' single deletes.
            u, slot = [], []
            for hub, pick in ((0, rng.permutation(deg)[:count]), (3, np.arange(count)),
                              (49, deg - 1 - np.arange(count))):
                u.append(np.full(len(pick), hub)), slot.append(pick)
            u.append(rng.integers(0, n, 40)), slot.append(rng.integers(0, 8, 40))
            if turn == 2:
                u.append(np.array([0, 0, 3, 49, 3])), slot.append(np.array([5, 5, 1 << 20, 0, 0xffffffff]))
            u = np.concatenate(u).astype(np.uint32)
            slot = np.concatenate(slot).astype(np.uint32)
            order = rng.permutation(len(u))
            bad = ex.delete(u[order], slot[order])
            if bad:
                with pytest.raises(BingoError) as e:
                    g.delete_batch(u[order], slot[order])
                assert e.value.status == 4 and f"({bad} deletes" in str(e.value)
            else:
                g.delete_batch(u[order], slot[order])
            _same(g, ex)
            k = 60
            ins = (rng.integers(0, 4, k).astype(np.uint32), rng.integers(0, n, k).astype(np.uint32),
                   rng.integers(1, 1 << 20, k).astype(np.uint32))
            assert np.array_equal(g.insert_batch(*ins), ex.insert(*ins))
            _same(g, ex)
        g.check()
        # Everything goes, in one batch per hub and order.
        for hub, order in ((0, slice(None)), (3, slice(None, None, -1))):
            all_slots = np.arange(g.dump()["ecnt"][hub], dtype=np.uint32)[order]
            bad = ex.delete(np.full(len(all_slots), hub, np.uint32), all_slots)
            try:
                g.delete_batch(np.full(len(all_slots), hub, np.uint32), all_slots)
                assert bad == 0
            except BingoError as e:
                assert e.status == 4 and bad
            _same(g, ex)
        g.check()
