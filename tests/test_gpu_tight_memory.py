"""Calls of a handle on a device with a few MB free: what the handle holds only for its next load makes room, so that
walks with host rows, update batches, the server, the tuner's copy of the store and restores run as on a handle that
holds nothing. Also batches after one that found no room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
N, M = 1500, 1_000_000  # some 667 edges per vertex: lists of 1024, which the batches below do not outgrow


class Hog:
    """Holds the device's free memory but for a few MB."""

    def __init__(self, leave=10 * MB):
        import torch
        self.held = []
        torch.cuda.synchronize()
        step = 1 << 40
        while step >= 2 * MB:
            free = torch.cuda.mem_get_info()[0] - leave
            step = min(step, free // (2 * MB) * 2 * MB)
            if step < 2 * MB:
                break
            try:
                self.held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                step //= 2

    def release(self):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def _edges(m, n, seed):
    rng = np.random.default_rng(seed)
    return (rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32),
            np.full(m, 4, np.uint32))


def _same(g, ex):
    a, b = g.dump(), ex.dump()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def _call(what, g, ex, tmp, small):
    """One call that takes some 20 to 40 MB on the large graph, checked against the oracle."""
    k = 3000 if small else 300_000
    n = g.n
    if what == "walk":
        starts = np.arange(k, dtype=np.uint32) % n
        got = g.walk(app=0, length=25, starts=starts, seed=3)  # staged in 32 MB (the next power of two)
        assert np.array_equal(got, ex.walk(0, 25, starts, seed=3))
    elif what == "insert":
        batch = _edges(k, n, 5)
        assert np.array_equal(g.insert_batch(*batch), ex.insert(*batch))
    elif what == "serve":
        g.serve_start(output_budget_bytes=(2 if small else 30) * MB, max_update_batch=1000)
        starts = np.arange(200, dtype=np.uint32) % n
        t, out = g.submit_walk(app=0, length=20, starts=starts, seed=4)
        g.serve_wait(t, timeout_us=20_000_000)
        g.serve_stop()
        assert np.array_equal(out, ex.walk(0, 20, starts, seed=4))
    elif what == "tune":
        rep = g.autotune(inserts=_edges(500, n, 6), repeats=1)
        assert rep["update_ms_start"] > 0, "the store was not copied"
        g.set_tuning(update_chunk=0)
    elif what == "restore":
        g.restore(tmp)


@pytest.mark.parametrize("what", ["walk", "insert", "serve", "tune", "restore"])
def test_kept_buffers_make_room(what, tmp_path):
    import torch
    from bingo_b200 import Graph
    from oracle import pyoracle as po
    assert torch.cuda.mem_get_info()[0] > 2 << 30
    path = str(tmp_path / "wide.bin")
    wide = 100_000
    exw = po.ExactGraph(wide)
    with Graph(device=0, node2vec=False) as g:  # also loads the kernels that the calls below need
        g.load_edges(*_edges(50_000, wide, 1), wide)
        exw.load(*_edges(50_000, wide, 1))
        g.save(path)
        _call(what, g, exw, path, True)
    with Graph(device=0, node2vec=False) as g:
        ex = po.ExactGraph(N)
        edges = _edges(M, N, 2)
        g.load_edges(*edges, N)
        ex.load(*edges)
        kept = g.stats()["scratch_bytes"]
        assert kept > 32 * MB, kept  # the load's scratch: what has to give way
        hog = Hog()
        try:
            _call(what, g, ex, path, False)
        finally:
            hog.release()
        if what == "restore":
            exr = po.ExactGraph(wide)
            exr.load(*_edges(50_000, wide, 1))
            _same(g, exr)
        else:
            assert g.stats()["scratch_bytes"] < kept + 40 * MB
            _same(g, ex)
        g.check()


def test_float_insert_after_load():
    from bingo_b200 import Graph
    src, dst, _ = _edges(M, N, 7)
    w = np.full(M, 0.5, np.float32)
    with Graph(device=0, node2vec=False, float_weights=True) as g:
        g.load_edges(src, dst, w, N)
        g.insert_batch(src[:100], dst[:100], w[:100])
        g.load_edges(src, dst, w, N)
        hog = Hog()
        try:
            slots = g.insert_batch(src[:300_000], dst[:300_000], w[:300_000])
        finally:
            hog.release()
        assert len(slots) == 300_000 and g.stats()["live_edges"] == M + 300_000
        g.check()


def test_batches_after_one_without_room():
    """Batches of growing size on a full device: refused whole from some size on; afterwards batches of every grouping
    form, and a load, run as if nothing had happened."""
    from bingo_b200 import BingoError, Graph
    from oracle import pyoracle as po
    with Graph(device=0, node2vec=False) as g:
        ex = po.ExactGraph(N)
        edges = _edges(M, N, 8)
        g.load_edges(*edges, N)
        ex.load(*edges)
        refused = 0
        hog = Hog(leave=4 * MB)
        try:
            for k in (110_000, 900_000, 1_100_000, 1_300_000, 1_500_000, 5_000_000, 120_000):
                batch = _edges(k, N, k)
                try:
                    slots = g.insert_batch(*batch)
                except BingoError as e:
                    assert e.name == "BINGO_ERR_CAPACITY"
                    refused += 1
                else:
                    assert np.array_equal(slots, ex.insert(*batch))
        finally:
            hog.release()
        assert refused >= 1
        for k in (120_000, 500, 140_000):
            batch = _edges(k, N, k + 1)
            assert np.array_equal(g.insert_batch(*batch), ex.insert(*batch))
        _same(g, ex)
        u = np.arange(110_000, dtype=np.uint32) % N
        slot = np.arange(110_000, dtype=np.uint32) // N
        g.delete_batch(u, slot)
        assert ex.delete(u, slot) == 0
        _same(g, ex)
        g.load_edges(*edges, N)
        fresh = po.ExactGraph(N)
        fresh.load(*edges)
        _same(g, fresh)
        g.check()
