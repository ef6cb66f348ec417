"""Performance cases of the walk engine: what is timed when its speed is compared between two versions.

Each case is a piece of work that a program using `bingo_b200.Graph` does in earnest, through the public calls:
walk queries of the four apps on resident graphs, streaming edge updates, batched programs that mix both, and the
build of a graph from an edge list. Graphs are R-MAT (a = 0.57, b = c = 0.19, edge factor 16, self-loops and repeated
edges dropped, like `bingo_b200.gen.rmat`), drawn on the GPU from the seed; weights, walk lengths, batch sizes and
parameters are those of bench.py's workloads. All results are vertex and slot ids (whole numbers); there is no
floating-point output, so there is no exact().
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bingo_b200 import BATCHED, DEEPWALK, NODE2VEC, PLAIN, PPR, SAMPLING, Graph, WalkJob

DEV = "cuda"
EDGE_FACTOR = 16
_stream = None
RESERVE = 8.0  # arena headroom a streaming program reserves, so that steady updates seldom reallocate
SETS = 3  # edge sets a streaming state turns over: one is absent, the others are in the graph


# ---------------------------------------------------------------------------------------------------- inputs
def _rmat(scale: int, gen: torch.Generator):
    """Sorted unique (src, dst) int64 keys of an R-MAT graph without self-loops."""
    m = EDGE_FACTOR << scale
    key = torch.zeros(m, dtype=torch.int64, device=DEV)
    for bit in range(scale):
        r = torch.rand(m, generator=gen, device=DEV)
        s = (r >= 0.76).to(torch.int64)                                   # lower half: c or d
        d = (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).to(torch.int64)    # right half: b or d
        key |= (s << (32 + bit)) | (d << bit)
    key = key[(key >> 32) != (key & 0xFFFFFFFF)]
    return torch.unique(key)


def _weights(kind: str, m: int, gen: torch.Generator):
    """int32 weights ("float": float32), of bench.py's distributions."""
    u = torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)
    if kind == "uniform10":      # uniform on [1, 1024]
        return (1 + u * 1024).to(torch.int32)
    if kind == "uniform16":      # uniform on [1, 65535]
        return (1 + u * 65535).to(torch.int32)
    if kind == "log20":          # log-uniform on [1, 2^20)
        return torch.exp2(u * 20).to(torch.int32).clamp_(1, (1 << 20) - 1)
    if kind == "zipf24":         # Zipf(1.2) on [1, 2^24): inverse of the continuous tail
        lo = 1.0 - (2.0 ** 24) ** -0.2
        return ((1.0 - u * lo) ** -5.0).to(torch.int32).clamp_(1, (1 << 24) - 1)
    if kind == "float":          # float weights, log-uniform on [2^-4, 2^10)
        return torch.exp2(u * 14 - 4).to(torch.float32)
    raise ValueError(kind)


def _split(key):
    return (key >> 32).to(torch.int32), (key & 0x7FFFFFFF).to(torch.int32)


def _graph(case: dict, gen: torch.Generator):
    key = _rmat(case["scale"], gen)
    src, dst = _split(key)
    return src.contiguous(), dst.contiguous(), _weights(case["weights"], key.numel(), gen)


def _open(case: dict) -> Graph:
    """A handle whose calls are ordered on the program's one compute stream, as in bench.py."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    g = Graph(device=torch.cuda.current_device(), node2vec=case["index"], synchronous=case["sync"],
              float_weights=case["weights"] == "float", arena_factor=RESERVE if "edges" in case else 2.0)
    g.set_stream(_stream.cuda_stream)
    return g


def _starts(src, k: int, gen: torch.Generator):
    """k uniform draws of vertices that have an out-edge."""
    walkable = torch.unique_consecutive(src)
    return walkable[torch.randint(walkable.numel(), (k,), generator=gen, device=DEV)].to(torch.int32)


def _churn(case: dict, src, dst, w, k: int, gen: torch.Generator):
    """SETS disjoint edge sets of k edges each: half taken from the graph's own edges (their sources follow the
    out-degree, as uniform deletes do), half new edges between uniform vertices (as uniform inserts are). Returns the
    edges to load, in random order, the sets, and where in the load each set begins; set 0 is left out of the load."""
    n = 1 << case["scale"]
    m = src.numel()
    own = k // 2
    pick = torch.randperm(m, generator=gen, device=DEV)
    new = k - own
    parts, sets, at = [], [], 0
    for _ in range(SETS):
        p = pick[at:at + own]
        at += own
        u = torch.randint(n, (new,), generator=gen, device=DEV, dtype=torch.int32)
        v = (u + torch.randint(1, n, (new,), generator=gen, device=DEV, dtype=torch.int32)) % n
        mix = torch.randperm(own + new, generator=gen, device=DEV)
        sets.append([torch.cat([src[p], u])[mix].contiguous(), torch.cat([dst[p], v])[mix].contiguous(),
                     torch.cat([w[p], _weights(case["weights"], new, gen)])[mix].contiguous()])
    rest = pick[at:]
    parts.append((src[rest], dst[rest], w[rest]))
    return [torch.cat(x).contiguous() for x in zip(*parts)], sets


# ---------------------------------------------------------------------------------------------------- cases
def _case(name, kind, scale, weights, index, sync, **more):
    c = {"kind": kind, "scale": scale, "weights": weights, "index": index, "sync": sync}
    c.update(more)
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # One-hop draws for one mini-batch of a sampler: the smallest call, where a call's own latency counts.
        _case("sample-4k", "walk", 18, "uniform10", True, True, app=SAMPLING, starts=4096, length=1),
        # One interactive query with numpy arrays in and out, the default of Graph.walk(): PPR from a few hundred
        # sources (bench.py's served queries: length 80, stop 0.15).
        _case("query-ppr-300-host", "host_query", 18, "uniform10", True, True, app=PPR, starts=300, length=80,
              stop=0.15),
        # A corpus of one DeepWalk per vertex on a small graph that lies in L2 (R-MAT 14, uniform weights).
        _case("deepwalk-16k", "walk", 14, "uniform10", False, False, app=DEEPWALK, starts=0, length=80),
        # The headline workload's walks: one DeepWalk of length 80 per vertex of R-MAT 20.
        _case("deepwalk-1m", "walk", 20, "log20", False, False, app=DEEPWALK, starts=0, length=80),
        # node2vec with the adjacency index and heavy-tailed weights (p = 0.5, q = 2, length 40), one per vertex.
        _case("node2vec-1m", "walk", 20, "zipf24", True, False, app=NODE2VEC, starts=0, length=40, p=0.5, q=2.0),
        # Random-walk-with-restart scores: 100K PPR walks from random sources with the reference's stop 0.0125,
        # float weights, an odd length.
        _case("ppr-100k-float", "walk", 19, "float", False, False, app=PPR, starts=100_003, length=101, stop=0.0125),
        # Sixteen walk jobs of all apps and sizes in one batched call (the jobs of bench.py's batched workload).
        _case("batch-16-jobs", "jobs", 20, "uniform16", True, False, jobs=16, lo=1000, hi=250_000),
        # Streaming updates: each pass inserts one edge set, deletes another by slot, and takes a short walk (two moves)
        # from every vertex just touched. A small batch on a default handle...
        _case("update-1k", "update", 16, "uniform16", True, True, edges=1000),
        # ... the headline workload's 50K + 50K batch ...
        _case("update-50k", "update", 20, "log20", False, False, edges=50_000),
        # ... and the node2vec workload's 500K + 500K, which also keeps the adjacency index.
        _case("update-500k-index", "update", 20, "zipf24", True, False, edges=500_000),
        # One phase of a batched program replayed as a CUDA graph: mixed walk jobs, an insert and a delete batch.
        _case("program-phase", "program", 20, "uniform16", True, False, jobs=8, lo=1000, hi=60_000, edges=20_000),
        # Build: a graph of 16 M edges from an edge list on the device, then a short walk (five moves) per vertex.
        _case("load-rmat20", "load", 20, "log20", False, True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    weights = rng.choice(["uniform10", "uniform16", "log20", "zipf24", "float"])
    sync = rng.random() < 0.5
    kind = rng.choice(["walk", "walk", "walk", "host_query", "jobs", "update", "update", "program", "load"])
    scale = rng.randint(12, 20)
    n = 1 << scale
    if kind == "walk":
        app = rng.choice([DEEPWALK, NODE2VEC, PPR, SAMPLING])
        c = _case(None, kind, scale, weights, app == NODE2VEC or rng.random() < 0.5, sync, app=app,
                  starts=log(200, n), length=1 if app == SAMPLING else rng.randint(5, 100))
        if app == NODE2VEC:
            c.update(length=min(c["length"], 60), p=rng.choice([0.25, 0.5, 1.0, 4.0]),
                     q=rng.choice([0.25, 1.0, 2.0, 4.0]))
        if app == PPR:
            c.update(stop=rng.choice([0.0125, 0.05, 0.15]))
        return c
    if kind == "host_query":
        app = rng.choice([DEEPWALK, PPR, SAMPLING])
        return _case(None, kind, scale, weights, False, True, app=app, starts=log(50, 3000),
                     length=1 if app == SAMPLING else rng.randint(5, 100), stop=0.15)
    if kind == "jobs":
        return _case(None, kind, scale, weights, True, sync, jobs=rng.randint(2, 24), lo=200, hi=log(500, n // 8))
    if kind == "program":
        return _case(None, kind, scale, weights if weights != "float" else "log20", True, False,
                     jobs=rng.randint(2, 16), lo=200, hi=log(500, n // 16), edges=log(200, n // 16))
    if kind == "update":
        return _case(None, kind, scale, weights, rng.random() < 0.5, sync, edges=log(200, n // 2))
    return _case(None, "load", scale, weights, rng.random() < 0.5, True)


def _job_sizes(case: dict):
    """(app, starts, length, p, q) of each job of a batched case: fixed by the case, not by the seed."""
    r = np.random.default_rng(case["jobs"] * 1_000_003 + case["hi"])
    out = []
    for j in range(case["jobs"]):
        k = int(np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]))))
        pq = [(a, b) for a in (0.25, 1.0, 4.0) for b in (0.25, 1.0, 4.0)][int(r.integers(0, 9))]
        out.append(([DEEPWALK, NODE2VEC, PPR][int(r.integers(0, 3))], k, int(r.integers(5, 201)), *pq))
    return out


def _jobs(case: dict, src, gen: torch.Generator, seed: int):
    jobs = []
    for j, (app, k, length, p, q) in enumerate(_job_sizes(case)):
        jobs.append(WalkJob(app=app, length=length, starts=_starts(src, k, gen), n_starts=k, job_id=j, seed=seed,
                            p=p, q=q, stop_prob=0.15, out=torch.empty((k, length), dtype=torch.int32, device=DEV)))
    return jobs


def prepare(case: dict, seed: int):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    src, dst, w = _graph(case, gen)
    n = 1 << case["scale"]
    g = _open(case)
    s = {"case": case, "g": g, "n": n, "seed": seed & 0x7FFFFFFF}
    kind = case["kind"]
    if kind == "load":
        order = torch.randperm(src.numel(), generator=gen, device=DEV)  # an edge list comes in no special order
        s.update(edges=(src[order], dst[order], w[order]), out=torch.empty((n, 6), dtype=torch.int32, device=DEV))
        torch.cuda.current_stream().synchronize()
        return s
    if kind in ("update", "program"):
        k = case["edges"]
        rest, sets = _churn(case, src, dst, w, k, gen)
        if kind == "program":
            s["jobs"] = _jobs(case, src, gen, s["seed"])
        torch.cuda.current_stream().synchronize()  # the handle's stream does not wait for torch's
        g.load_edges(*rest, n)
        slots = [torch.zeros(k, dtype=torch.int32, device=DEV) for _ in sets]
        torch.cuda.current_stream().synchronize()
        for b in range(1, SETS):
            g.insert_batch(*sets[b], out_slots=slots[b])
        g.sync()
        s.update(sets=sets, slots=slots, turn=0, out=torch.empty((k, 3), dtype=torch.int32, device=DEV))
        torch.cuda.current_stream().synchronize()
        return s
    torch.cuda.current_stream().synchronize()
    g.load_edges(src, dst, w, n)
    if kind == "jobs":
        s["jobs"] = _jobs(case, src, gen, s["seed"])
    elif kind == "host_query":
        s["starts"] = _starts(src, case["starts"], gen).cpu().numpy().astype(np.uint32)
    else:
        k = case["starts"]
        if k:
            s["starts"] = _starts(src, k, gen)
        k = k or n
        shape = (k,) if case["app"] == SAMPLING else (k, case["length"])
        s.update(k=k, out=torch.empty(shape, dtype=torch.int32, device=DEV))
    torch.cuda.current_stream().synchronize()
    return s


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind == "walk":
        g.walk(app=case["app"], length=case["length"], starts=s.get("starts"), n_starts=s["k"], seed=s["seed"],
               p=case.get("p", 0.5), q=case.get("q", 2.0), stop_prob=case.get("stop", 0.0125), mode=PLAIN,
               out=s["out"])
        return s["out"]
    if kind == "host_query":
        return g.walk(app=case["app"], length=case["length"], starts=s["starts"], seed=s["seed"],
                      stop_prob=case["stop"])
    if kind == "jobs":
        g.walk_jobs(s["jobs"], mode=BATCHED)
        return [j.out for j in s["jobs"]]
    if kind == "load":
        g.load_edges(*s["edges"], s["n"])
        g.walk(app=DEEPWALK, length=6, n_starts=s["n"], seed=s["seed"], out=s["out"])
        return s["out"]
    # A turn of a streaming state: the absent set comes in, the next one goes out.
    i, d = s["turn"] % SETS, (s["turn"] + 1) % SETS
    s["turn"] += 1
    ins, dele = s["sets"][i], s["sets"][d]
    if kind == "update":
        g.insert_batch(*ins, out_slots=s["slots"][i])
        g.delete_batch(dele[0], s["slots"][d])
        g.walk(app=DEEPWALK, length=3, starts=dele[0], seed=s["seed"], job_id=s["turn"], out=s["out"])
        return {"slots": s["slots"][i], "walks": s["out"]}
    # Program: the walks, the insert and the delete without a host wait between them.
    g.run([("walk", s["jobs"]), ("insert", *ins, s["slots"][i]), ("delete", dele[0], s["slots"][d]),
           ("walk", [WalkJob(app=DEEPWALK, length=3, starts=dele[0], n_starts=dele[0].numel(), seed=s["seed"],
                             job_id=s["turn"], out=s["out"])])])
    return {"rows": [j.out for j in s["jobs"]], "slots": s["slots"][i], "walks": s["out"]}


# ---------------------------------------------------------------------------------------------------- work
def _step_share(scale: int) -> float:
    """Share of a row's positions that hold a move when walks start at every vertex: many R-MAT vertices have no
    out-edge (0.81 of them at scale 14 and 0.38 at scale 20, measured)."""
    return min(0.85, max(0.35, 0.81 - (scale - 14) * 0.072))


def _walk_bytes(app, k, length, scale, stop, everywhere):
    """Rows written once, starts read, and per move: vertex 8 B, alias slot 8 B, group 4 B, member 8 B; node2vec: 1.87
    proposals of 28 B and 1.9 adjacency lookups of 8 B per move."""
    if app == SAMPLING:
        return k * (4 + 4 + 28)
    share = _step_share(scale) if everywhere else min(0.9, 1.4 * _step_share(scale))
    moves = length * share
    if app == PPR:
        moves = min(moves, 1.0 / stop)
    per = 1.87 * 28 + 1.9 * 8 if app == NODE2VEC else 28
    return k * (4 * length + (0 if everywhere else 4) + per * moves)


def _update_bytes(weights, k, index):
    """Per edge, p = set bits of a weight and m = groups of a vertex: insert 12 B read, 8 B slot record, 8 B per member,
    delete 16 B and 16 B per member, and 2 x 16 B of alias table per group of each touched vertex; the index 16 B."""
    p, m = {"uniform10": (5, 8), "uniform16": (8, 13), "log20": (5.6, 11), "zipf24": (2.6, 6), "float": (12, 16)}[weights]
    return k * (20 + 8 * p + 32 * m + 20 + 16 * p + 32 * m + (32 if index else 0))


def work(case: dict):
    kind, scale = case["kind"], case["scale"]
    n = 1 << scale
    b = 0.0
    if kind in ("walk", "host_query"):
        b = _walk_bytes(case["app"], case["starts"] or n, case["length"], scale, case.get("stop", 0.0125),
                        not case["starts"])
    elif kind == "load":
        m = EDGE_FACTOR * n * 0.96
        p, groups = {"uniform10": (5, 7), "uniform16": (8, 10), "log20": (5.6, 8), "zipf24": (2.6, 5),
                     "float": (12, 12)}[case["weights"]]
        b = m * (12 + 16 + 12 * p + (32 if case["index"] else 0)) + n * (16 + 48 + 256 + 32 * groups * 0.6 + 24 + 28 * 2)
    if kind in ("jobs", "program"):
        b += sum(_walk_bytes(app, k, length, scale, 0.15, False) for app, k, length, _, _ in _job_sizes(case))
    if kind in ("update", "program"):
        b += _update_bytes(case["weights"], case["edges"], case["index"]) + case["edges"] * (16 + 2 * 28)
    return {"bytes": b, "flops": 0}
