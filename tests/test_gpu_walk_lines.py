"""Walk rows at the edges of the output lines they are collected in, and node2vec steps that take many trials: rows
that start and end anywhere in a 128-byte line, launches from one walk to more than the resident lanes, every app in
one table. Compared with the CPU oracle row for row; memory around the rows must stay untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = -77


@pytest.fixture(scope="module")
def pair():
    from bingo_b200 import Graph, gen
    from oracle import pyoracle as po
    n = 1 << 11
    src, dst = gen.rmat(11, 12, seed=31)
    w = gen.weights(len(src), gen.W_LOGUNIFORM, 1, 1 << 20, seed=32)
    g, ex = Graph(device=0), po.ExactGraph(n)
    g.load_edges(src, dst, w, n)
    ex.load(src, dst, w)
    yield g, ex, n
    g.close()


def _rows(torch, k, length, shift):
    """A device buffer with k rows of `length` at a 32-byte offset `shift`, guard values all around."""
    buf = torch.full((shift * 8 + k * length + 64,), GUARD, dtype=torch.int32, device="cuda")
    return buf, buf[shift * 8:shift * 8 + k * length].view(k, length)


def _check(buf, rows, want, shift):
    got = rows.cpu().numpy()
    assert np.array_equal(got, want)
    flat = buf.cpu().numpy()
    assert (flat[:shift * 8] == GUARD).all() and (flat[shift * 8 + got.size:] == GUARD).all()


@pytest.mark.parametrize("length", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 100])
@pytest.mark.parametrize("app", [0, 1, 2])
def test_rows_at_line_edges(pair, app, length):
    import torch
    g, ex, n = pair
    rng = np.random.default_rng(100 * app + length)
    for k, shift in ((1, 0), (33, 1), (300, 3), (2048, 2)):
        starts = rng.integers(0, n, k).astype(np.uint32)
        flags = 1 if app == 2 and k == 300 else 0  # PPR tail: the last position is rewritten
        buf, rows = _rows(torch, k, length, shift)
        dev = torch.from_numpy(starts.view(np.int32)).cuda()
        torch.cuda.synchronize()
        g.walk(app=app, length=length, starts=dev, seed=5, job_id=k, p=0.5, q=2.0, stop_prob=0.1, flags=flags,
               out=rows)
        want = ex.walk(app, length, starts, seed=5, job_id=k, p=0.5, q=2.0, stop=0.1, flags=flags)
        _check(buf, rows, want, shift)


@pytest.mark.parametrize("p,q", [(0.25, 4.0), (4.0, 4.0), (4.0, 0.25), (0.01, 8.0), (1.0, 64.0)])
@pytest.mark.parametrize("k", [1, 3, 17, 40, 5000, 200_000])
def test_many_trials(pair, p, q, k):
    """Trials per step from one to dozens, with warps that hold one walk and full ones."""
    g, ex, n = pair
    starts = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    length = 21 if k < 10_000 else 6
    t0 = g.stats()
    out = g.walk(app=1, length=length, starts=starts, seed=9, job_id=k, p=p, q=q)
    t1 = g.stats()
    assert np.array_equal(out, ex.walk(1, length, starts, seed=9, job_id=k, p=p, q=q))
    moves = int((out[:, 1:] >= 0).sum())
    assert t1["walk_steps"] - t0["walk_steps"] == moves
    second = int((out[:, 2:] >= 0).sum())  # every second-order move drew a proposal or returned by its region
    assert t1["walk_trials"] - t0["walk_trials"] >= (second if p >= 1 else 0)


def test_mixed_tables(pair):
    """Every app in one launch, from few walks per job to more than a warp claims at once."""
    import torch
    from bingo_b200 import BATCHED, WalkJob
    g, ex, n = pair
    rng = np.random.default_rng(8)
    for sizes in ((1, 2, 1, 3), (40, 1, 700, 33), (9000, 5000, 1, 60_000)):
        jobs, want = [], []
        for j, (k, app) in enumerate(zip(sizes * 2, (1, 0, 2, 3, 2, 1, 0, 1))):
            length = int(rng.integers(1, 50))
            starts = rng.integers(0, n, k).astype(np.uint32)
            p, q = float(rng.choice([0.25, 1, 4])), float(rng.choice([0.25, 1, 4]))
            shape = (k,) if app == 3 else (k, length)
            jobs.append(WalkJob(app=app, length=length, starts=torch.from_numpy(starts.view(np.int32)).cuda(),
                                n_starts=k, job_id=j, seed=3, p=p, q=q, stop_prob=0.2,
                                out=torch.full(shape, GUARD, dtype=torch.int32, device="cuda")))
            want.append(ex.walk(app, length, starts, seed=3, job_id=j, p=p, q=q, stop=0.2))
        torch.cuda.synchronize()
        g.walk_jobs(jobs, mode=BATCHED)
        for j, x in zip(jobs, want):
            assert np.array_equal(j.out.cpu().numpy(), x.reshape(j.out.shape))
