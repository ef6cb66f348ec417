"""node2vec jobs of their own around the sizes at which a launch stops fitting its lanes, and small ones, for p and q
whose steps take one trial, a few and many: rows against the oracle; the counts of trials and lookups do not depend on
how the walks are launched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    from bingo_b200 import Graph, gen
    from oracle import pyoracle as po
    n = 1 << 12
    src, dst = gen.rmat(12, 10, seed=8)
    w = gen.weights(len(src), gen.W_UNIFORM, 1, 1 << 16, seed=9)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    with Graph(device=0, node2vec=True) as g:
        g.load_edges(src, dst, w, n)
        yield g, ex, n


@pytest.mark.parametrize("p,q", [(1.0, 1.0), (0.25, 0.25), (4.0, 0.5), (0.5, 2.0), (4.0, 8.0)])
def test_rows_at_every_size(graph, p, q):
    import torch
    g, ex, n = graph
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 256
    for k, length in ((1, 50), (31, 9), (64, 20), (65, 20), (257, 33), (lanes // 4 - 1, 5), (lanes // 2 + 1, 5),
                      (lanes - 1, 4), (lanes, 4), (lanes + 1, 4), (2 * lanes + 77, 3)):
        starts = (np.arange(k, dtype=np.uint64) * 2654435761 % n).astype(np.uint32)
        out = torch.full((k, length), -9, dtype=torch.int32, device="cuda")
        g.walk(app=1, length=length, starts=torch.from_numpy(starts.view(np.int32)).cuda(), seed=k, p=p, q=q, out=out)
        assert np.array_equal(out.cpu().numpy(), ex.walk(1, length, starts, seed=k, p=p, q=q)), (k, length)


def test_counts_do_not_depend_on_the_launch(graph):
    """The same walks in one job, in two, and in a table: equal proposals and lookups."""
    import torch
    from bingo_b200 import BATCHED, PLAIN, WalkJob
    g, ex, n = graph
    k = 6000
    starts = torch.from_numpy((np.arange(k) * 7919 % n).astype(np.int32)).cuda()
    counts = []
    for p, q in ((1.0, 1.0), (0.25, 0.25), (0.5, 3.0)):
        for mode in (PLAIN, BATCHED):
            for chunk in (0, 1, 32):
                g.set_tuning(walk_chunk=chunk)
                s0 = g.stats()
                out = torch.empty((k, 12), dtype=torch.int32, device="cuda")
                g.walk_jobs([WalkJob(app=1, length=12, starts=starts, n_starts=k, seed=3, p=p, q=q, out=out)], mode=mode)
                s1 = g.stats()
                counts.append((p, q, s1["walk_trials"] - s0["walk_trials"], s1["walk_probes"] - s0["walk_probes"],
                               s1["walk_steps"] - s0["walk_steps"]))
    g.set_tuning(walk_chunk=0)
    assert len(set(counts)) == 3
