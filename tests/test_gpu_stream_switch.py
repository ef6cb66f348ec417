"""Walk launches of one asynchronous handle that overlap on two streams share its work counters: whatever the
overlapping calls leave there, every later walk is whole. Also walks captured by the caller and replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(scale, seed):
    from bingo_b200 import gen
    from oracle import pyoracle as po
    n = 1 << scale
    src, dst = gen.rmat(scale, 8, seed=seed)
    w = gen.weights(len(src), gen.W_UNIFORM, 1, 1 << 16, seed=seed + 1)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    return n, (src, dst, w), ex


@pytest.mark.parametrize("small", [1, 300, 9000])
def test_walks_after_overlapping_ones(small):
    """Plain walks of unequal sizes in flight on two streams (their own rows are the caller's to order), then walks of
    every form on either stream, each against the oracle."""
    import torch
    from bingo_b200 import BATCHED, PLAIN, Graph, WalkJob
    n, edges, ex = _graph(12, 31)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    many = torch.arange(n, dtype=torch.int32, device="cuda").repeat(60)
    few = torch.arange(small, dtype=torch.int32, device="cuda") % n
    out = torch.empty((len(many), 40), dtype=torch.int32, device="cuda")
    out2 = torch.empty((small, 40), dtype=torch.int32, device="cuda")
    want = ex.walk(0, 40, np.arange(n, dtype=np.uint32), seed=9)
    rows = torch.empty((n, 40), dtype=torch.int32, device="cuda")
    with Graph(device=0, synchronous=False, node2vec=False) as g:
        g.set_stream(a.cuda_stream)
        g.load_edges(*edges, n)
        torch.cuda.synchronize()
        for turn in range(4):
            for _ in range(3):
                g.walk(app=0, length=40, starts=many, seed=3, out=out)
                g.set_stream(b.cuda_stream)
                for _ in range(5):
                    g.walk(app=0, length=40, starts=few, seed=4, out=out2)
                g.set_stream(a.cuda_stream)
            torch.cuda.synchronize()
            if turn % 2:
                g.set_stream(b.cuda_stream)
            for form in (lambda j: g.walk_jobs(j, mode=PLAIN), lambda j: g.walk_jobs(j, mode=BATCHED),
                         lambda j: g.run([("walk", j)]), lambda j: g.run([("walk", j)], graph=True)):
                rows.fill_(-9)
                torch.cuda.synchronize()
                form([WalkJob(app=0, length=40, n_starts=n, seed=9, out=rows)])
                torch.cuda.synchronize()
                assert np.array_equal(rows.cpu().numpy(), want)
            g.set_stream(a.cuda_stream)


def test_captured_walk_replayed_between_calls():
    import torch
    from bingo_b200 import Graph
    n, edges, ex = _graph(10, 41)
    s = torch.cuda.Stream()
    rows = torch.empty((n, 12), dtype=torch.int32, device="cuda")
    other = torch.empty((700, 12), dtype=torch.int32, device="cuda")
    want = ex.walk(0, 12, np.arange(n, dtype=np.uint32), seed=5)
    want2 = ex.walk(0, 12, np.arange(700, dtype=np.uint32), seed=6)
    with Graph(device=0, synchronous=False) as g:
        g.load_edges(*edges, n)
        g.walk(app=0, length=12, n_starts=n, seed=5, out=rows)
        g.sync()
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            g.set_stream(torch.cuda.current_stream().cuda_stream)
            g.walk(app=0, length=12, n_starts=n, seed=5, out=rows)
        g.set_stream(s.cuda_stream)
        for _ in range(3):
            with torch.cuda.stream(s):
                rows.fill_(-9)
                other.fill_(-9)
                graph.replay()
                g.walk(app=0, length=12, n_starts=700, seed=6, out=other)
                graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(rows.cpu().numpy(), want)
            assert np.array_equal(other.cpu().numpy(), want2)
