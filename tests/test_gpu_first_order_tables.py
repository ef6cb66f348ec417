"""Job tables without node2vec jobs (their own kernel) and with them, one app or several, in every call that takes a
table: rows against the oracle. A captured program replayed with jobs of other apps follows the change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DW, N2V, PPR, ONE = 0, 1, 2, 3
TAIL = 1  # BINGO_WALK_PPR_TAIL


def _graph(index):
    from bingo_b200 import Graph, gen
    from oracle import pyoracle as po
    n = 1 << 12
    src, dst = gen.rmat(12, 8, seed=5)
    w = gen.weights(len(src), gen.W_UNIFORM, 1, 1 << 16, seed=6)
    ex = po.ExactGraph(n)
    ex.load(src, dst, w)
    g = Graph(device=0, node2vec=index)
    g.load_edges(src, dst, w, n)
    return g, ex, n


def _jobs(spec, n, seed):
    """(app, length, walks, flags) -> jobs with device outputs."""
    import torch
    from bingo_b200 import WalkJob
    out = []
    for j, (app, length, k, flags) in enumerate(spec):
        rng = np.random.default_rng(seed + j)
        starts = rng.integers(0, n, k).astype(np.uint32)
        shape = (k,) if app == ONE else (k, length)
        out.append(WalkJob(app=app, length=length, starts=torch.from_numpy(starts.view(np.int32)).cuda(), n_starts=k,
                           job_id=j, seed=seed, flags=flags, p=0.5, q=2.0, stop_prob=0.1,
                           out=torch.full(shape, -9, dtype=torch.int32, device="cuda")))
    return out


def _noalloc(g, jobs):
    from bingo_b200 import lib
    arr = g._job_array(jobs, [])
    assert lib().bingo_walk_noalloc(g.handle, arr, len(jobs)) == 0


def _same(jobs, ex):
    for j in jobs:
        want = ex.walk(j.app, j.length, j.starts.cpu().numpy().view(np.uint32), seed=j.seed, job_id=j.job_id, p=j.p,
                       q=j.q, stop=j.stop_prob, flags=j.flags)
        assert np.array_equal(j.out.cpu().numpy().reshape(want.shape), want), (j.app, j.length, j.n_starts, j.flags)


SPECS = {
    "deepwalk": [(DW, 40, 3000, 0), (DW, 7, 1, 0), (DW, 1, 500, 0), (DW, 33, 2111, 0)],
    "ppr": [(PPR, 20, 900, 0), (PPR, 1, 300, TAIL), (PPR, 6, 5000, TAIL), (PPR, 65, 31, 0)],
    "one hop": [(ONE, 1, 70000, 0), (ONE, 1, 1, 0), (ONE, 1, 4097, 0)],
    "first order": [(DW, 80, 700, 0), (ONE, 1, 3000, 0), (PPR, 9, 2500, 0), (PPR, 2, 100, TAIL), (DW, 3, 33, 0),
                    (PPR, 80, 1, 0), (ONE, 1, 5, 0)],
    "many short": [(PPR, 8, 200_000, 0), (ONE, 1, 100_000, 0), (DW, 2, 50_000, 0)],
    "with node2vec": [(DW, 40, 900, 0), (N2V, 20, 800, 0), (PPR, 30, 1200, 0), (ONE, 1, 64, 0)],
}


@pytest.mark.parametrize("index", [False, True])
@pytest.mark.parametrize("name", list(SPECS))
def test_tables(name, index):
    from bingo_b200 import BATCHED
    if name == "with node2vec" and not index:
        pytest.skip("needs the index")
    g, ex, n = _graph(index)
    with g:
        for form in (lambda j: g.walk_jobs(j, mode=BATCHED), lambda j: g.run([("walk", j)], graph=False),
                     lambda j: g.run([("walk", j)], graph=True), lambda j: _noalloc(g, j)):
            jobs = _jobs(SPECS[name], n, 11)
            form(jobs)
            _same(jobs, ex)
        g.set_tuning(walk_chunk=5)
        jobs = _jobs(SPECS[name], n, 12)
        g.walk_jobs(jobs, mode=BATCHED)
        _same(jobs, ex)


def test_program_whose_jobs_change_app():
    g, ex, n = _graph(True)
    sizes = [(20, 900), (7, 300), (33, 2000)]
    order = [(DW, DW, DW), (PPR, DW, PPR), (DW, N2V, DW), (N2V, N2V, N2V), (DW, PPR, DW), (DW, DW, N2V)]
    with g:
        for turn, apps in enumerate(order * 2):
            jobs = _jobs([(a, length, k, 0) for a, (length, k) in zip(apps, sizes)], n, 20 + turn)
            g.run([("walk", jobs)], graph=True)
            _same(jobs, ex)
