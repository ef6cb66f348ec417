"""A handle that loads a smaller graph after a larger one holds about what a handle that loaded only the smaller one
does, and computes the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.55, 0.8])
def test_memory_after_a_smaller_load(share):
    import torch
    from bingo_b200 import Graph
    n, m = 30_000, 6_000_000
    rng = np.random.default_rng(1)
    src, dst = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    w = rng.integers(1, 1 << 16, m).astype(np.uint32)
    small = int(m * share)

    def held(sizes):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with Graph(device=0, node2vec=False) as g:
            for k in sizes:
                g.load_edges(src[:k], dst[:k], w[:k], n)
            used = before - torch.cuda.mem_get_info()[0]
            rows = g.walk(app=0, length=20, n_starts=2000, seed=3)
            return used, rows

    held([1000])  # kernels and their memory are in place
    alone, rows = held([small])
    after, rows2 = held([m, small])
    assert np.array_equal(rows, rows2)
    # A sixteenth and 1 MB per buffer (a dozen) are kept at most; allocations come in pages of 2 MB.
    assert after <= alone * 17 / 16 + 12 * (3 << 20), (alone >> 20, after >> 20)
