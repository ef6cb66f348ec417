"""Delete batches in device memory with vertex ids >= n, in orders that make many more segment heads than the graph
has vertices: refused whole, in every grouping form, by the call and by a program, and the handle goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 300])
@pytest.mark.parametrize("k", [60, 4000, 98_304, 98_305, 400_000])
def test_ids_past_n_in_long_runs(n, k):
    import torch
    from bingo_b200 import BingoError, Graph
    from oracle import pyoracle as po
    rng = np.random.default_rng(n + k)
    src = np.repeat(np.arange(n, dtype=np.uint32), 40)
    dst, w = rng.integers(0, n, len(src)).astype(np.uint32), rng.integers(1, 1 << 16, len(src)).astype(np.uint32)
    bits = max(1, int(n - 1).bit_length())
    at = np.arange(k, dtype=np.uint64)
    batches = [
        (at % 24) << bits,                          # equal in the bits that are sorted, another id at each place
        (at // 25 + 1) << bits,                     # a new id every 25 places
        np.where(at % 2 == 0, 0, 1 << bits),        # valid ids among them
        rng.integers(0, 1 << 31, k, dtype=np.uint64),
    ]

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x.astype(np.uint32).view(np.int32))).cuda()

    with Graph(device=0, node2vec=True) as g:
        ex = po.ExactGraph(n)
        g.load_edges(src, dst, w, n)
        ex.load(src, dst, w)
        want = ex.dump()
        slots = dev(at % 40)
        for u in batches:
            for call in (lambda: g.delete_batch(dev(u), slots), lambda: g.run([("delete", dev(u), slots)])):
                with pytest.raises(BingoError) as e:
                    call()
                assert e.value.status == 2
                g.sync()
        got = g.dump()
        for c in want:
            assert np.array_equal(got[c], want[c]), c
        u, slot = np.repeat(np.arange(n, dtype=np.uint32), 30), np.tile(np.arange(30, dtype=np.uint32), n)
        g.delete_batch(u, slot)
        assert ex.delete(u, slot) == 0
        got, want = g.dump(), ex.dump()
        for c in want:
            assert np.array_equal(got[c], want[c]), c
        g.check()
