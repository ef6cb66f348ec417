"""What a handle keeps between calls: graph buffers and load scratch over loads of other sizes, the error flag that
spares a status copy, and the walk work counters that a launch leaves zeroed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(scale, seed, weights=1 << 16):
    from bingo_b200 import gen
    src, dst = gen.rmat(scale, 8, seed=seed)
    return 1 << scale, src, dst, gen.weights(len(src), gen.W_UNIFORM, 1, weights, seed=seed + 1)


def _same(g, ex):
    a, b = g.dump(), ex.dump()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("index", [True, False])
def test_loads_of_other_sizes(index):
    """Larger, smaller, equal and empty graphs in turn on one handle, with updates and walks between."""
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    with Graph(device=0, node2vec=index) as g:
        for turn, scale in enumerate((9, 12, 12, 5, 14, 6, 10)):
            n, src, dst, w = _case(scale, 50 + turn)
            ex = po.ExactGraph(n)
            g.load_edges(src, dst, w, n)
            ex.load(src, dst, w)
            _same(g, ex)
            k = min(len(src), 700)
            slots = g.insert_batch(dst[:k], src[:k], w[:k])
            assert np.array_equal(slots, ex.insert(dst[:k], src[:k], w[:k]))
            g.delete_batch(dst[:k], slots)
            ex.delete(dst[:k], slots)
            _same(g, ex)
            starts = np.arange(n, dtype=np.uint32)
            assert np.array_equal(g.walk(app=0, length=9, starts=starts, seed=turn),
                                  ex.walk(0, 9, starts, seed=turn))
            st = g.stats()
            assert st["arena_used"] <= st["arena_bytes"]
        empty = np.zeros(0, np.uint32)
        g.load_edges(empty, empty, empty, 10)
        assert g.stats()["live_edges"] == 0


def test_rejected_load_then_good():
    import torch
    from bingo_b200 import BingoError, Graph
    from oracle import pyoracle as po
    n, src, dst, w = _case(10, 3)
    dev = [torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst, w)]
    with Graph(device=0) as g:
        bad = dev[2].clone()
        bad[5] = 0
        torch.cuda.synchronize()
        g.load_edges(dev[0], dev[1], dev[2], n)
        with pytest.raises(BingoError) as e:
            g.load_edges(dev[0], dev[1], bad, n)
        assert e.value.status == 3
        with pytest.raises(BingoError) as e:  # the failed load left no graph
            g.walk(app=0, length=3, starts=np.zeros(1, np.uint32))
        assert e.value.status == 7
        g.load_edges(dev[0], dev[1], dev[2], n)
        ex = po.ExactGraph(n)
        ex.load(src, dst, w)
        _same(g, ex)


@pytest.mark.parametrize("synchronous", [True, False])
def test_errors_are_reported_once(synchronous):
    """Every device-detected error reaches the host, once, and later calls are clean."""
    import torch
    from bingo_b200 import BingoError, Graph
    n, src, dst, w = _case(8, 9)
    with Graph(device=0, synchronous=synchronous) as g:
        g.load_edges(src, dst, w, n)
        bad_start = torch.full((4,), n + 5, dtype=torch.int32, device="cuda")
        good = torch.zeros(4, dtype=torch.int32, device="cuda")
        out = torch.zeros((4, 8), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

        def fails(status, call):
            with pytest.raises(BingoError) as e:
                call()
                g.sync()
            assert e.value.status == status

        for _ in range(3):
            fails(2, lambda: g.walk(app=0, length=8, starts=bad_start, out=out))
            g.walk(app=0, length=8, starts=good, out=out)
            g.sync()
            fails(4, lambda: g.delete_batch(np.zeros(2, np.uint32), np.full(2, 1 << 30, np.uint32)))
            g.sync()
            fails(2, lambda: g.insert_batch(bad_start, good, torch.ones_like(good), return_slots=False))
            g.sync()


def test_counters_after_every_shape():
    """Launches of many shapes in a row, plain, batched, as programs and without allocation: each finds its work
    counter zeroed by the one before."""
    import torch
    from bingo_b200 import BATCHED, PLAIN, Graph, WalkJob
    from oracle import pyoracle as po
    n, src, dst, w = _case(9, 21)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    rng = np.random.default_rng(2)
    with Graph(device=0) as g:
        g.load_edges(src, dst, w, n)
        for turn, jobs_n in enumerate((1, 3, 70, 2, 1)):
            jobs, want = [], []
            for j in range(jobs_n):
                app, k = int(rng.integers(0, 4)), int(rng.integers(1, 400))
                starts = rng.integers(0, n, k).astype(np.uint32)
                shape = (k,) if app == 3 else (k, 12)
                jobs.append(WalkJob(app=app, length=12, starts=torch.from_numpy(starts.view(np.int32)).cuda(),
                                    n_starts=k, job_id=j, seed=turn, out=torch.zeros(shape, dtype=torch.int32, device="cuda")))
                want.append(ex.walk(app, 12, starts, seed=turn, job_id=j))
            torch.cuda.synchronize()
            for form in (lambda: g.walk_jobs(jobs, mode=PLAIN), lambda: g.walk_jobs(jobs, mode=BATCHED),
                         lambda: g.run([("walk", jobs), ("walk", jobs[:1])]),
                         lambda: g.run([("walk", jobs), ("walk", jobs[:1])])):
                for j in jobs:
                    j.out.fill_(-9)
                torch.cuda.synchronize()
                form()
                for j, x in zip(jobs, want):
                    assert np.array_equal(j.out.cpu().numpy(), x.reshape(j.out.shape))


def test_load_after_a_stream_change():
    """A load while walks on the handle's earlier stream may still run: their rows and the new graph are both right."""
    import torch
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    n, src, dst, w = _case(12, 31)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    dev = [torch.from_numpy(x.view(np.int32)).cuda() for x in (src, dst, w)]
    rev = [dev[1], dev[0], dev[2]]
    ex2 = po.ExactGraph(n)
    ex2.load(dst, src, w)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    starts = torch.arange(n, dtype=torch.int32, device="cuda").repeat(20)
    want = ex.walk(0, 40, starts.cpu().numpy().astype(np.uint32), seed=3)
    want2 = ex2.walk(0, 40, np.arange(n, dtype=np.uint32), seed=4)
    for _ in range(3):
        with Graph(device=0, synchronous=False, node2vec=False) as g:
            out = torch.empty((len(starts), 40), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            g.set_stream(a.cuda_stream)
            g.load_edges(*dev, n)
            for _ in range(4):
                g.walk(app=0, length=40, starts=starts, seed=3, out=out)
            g.set_stream(b.cuda_stream)
            g.load_edges(*rev, n)
            out2 = torch.empty((n, 40), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            g.walk(app=0, length=40, n_starts=n, seed=4, out=out2)
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)
            assert np.array_equal(out2.cpu().numpy(), want2)


def test_loads_while_another_thread_captures():
    """One handle loads again and again while another captures programs of changing shape on its own thread."""
    import threading

    import torch
    from bingo_b200 import Graph, WalkJob
    from oracle import pyoracle as po
    n, src, dst, w = _case(9, 41)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    failed = []

    def programs():
        try:
            with Graph(device=0, synchronous=False) as g:
                g.load_edges(src, dst, w, n)
                for turn in range(60):
                    k = 20 + turn
                    out = torch.zeros((k, 10), dtype=torch.int32, device="cuda")
                    g.sync()
                    g.run([("walk", [WalkJob(app=0, length=10, n_starts=k, seed=turn, out=out)])])
                    g.sync()
                    if not np.array_equal(out.cpu().numpy(), ex.walk(0, 10, np.arange(k, dtype=np.uint32), seed=turn)):
                        failed.append(turn)
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    t = threading.Thread(target=programs)
    t.start()
    with Graph(device=0) as g:
        for turn in range(40):
            g.load_edges(src, dst, w, n)
        _same(g, ex)
    t.join()
    assert not failed, failed[:3]
