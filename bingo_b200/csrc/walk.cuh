// Walk-step sampler and the per-app walk loops. Replaces NodeData::sample
// (include/Bingo.cuh:220-267) and the loops of deepwalkKernel, node2vecKernel,
// pprKernel and samplingKernel (include/operation.cuh:252-368, :407-430).
//
// One step is at most three dependent loads: the 16 B VertexRec of the
// current vertex, the 32 B AliasRec of the drawn slot (which names both
// candidate groups: member-list base and count, or for a one-member group the
// member itself), and the 4 B member id (skipped for a one-member group). All
// go through the read-only path: the store does not change during a walk
// phase.
#pragma once
#include "common.cuh"
#include "store.cuh"

namespace bingo {

constexpr uint32_t kMaxNode2vecTrials = 1u << 16;
constexpr uint32_t kMaxPprSteps = 1u << 20;
constexpr uint32_t kWalkPprTail = 1u;

enum AppId : int { APP_DEEPWALK = 0, APP_NODE2VEC = 1, APP_PPR = 2, APP_SAMPLING = 3 };
// Kernels of job tables: jobs of any app, and jobs that are not node2vec.
constexpr int APP_MIXED = -1, APP_FIRST = -2;

// One walk job as the kernels see it (starts/out are device pointers).
struct WalkJobDev {
  int32_t app;
  uint32_t L;
  const uint32_t* starts;  // null: first + walk index
  unsigned long long n;
  uint32_t first;
  uint32_t job;
  uint32_t k0, k1;  // Philox key (seed)
  uint32_t flags;
  uint32_t seq;  // serving ring: the job's sequence number (0 elsewhere)
  unsigned long long thr_ret, thr_in, thr_out, thr_stop;  // 33-bit acceptance thresholds
  double ret_excess;  // node2vec: (1/p) / max(1, 1/q) - 1 when positive, else 0
  int32_t* out;
};

// p in [0, 1] -> 33-bit threshold floor(p * 2^32) (2^32 = always); the same
// formula as the host side, with IEEE-rounded operations.
__device__ __forceinline__ unsigned long long prob_threshold_dev(double p) {
  if (!(p > 0.0)) return 0ull;
  if (p >= 1.0) return 1ull << 32;
  const double t = floor(__dmul_rn(p, 4294967296.0));
  return t >= 4294967296.0 ? (1ull << 32) : (unsigned long long)t;
}

struct WalkView {
  uint32_t n;
  const VertexRec* __restrict__ vrec;
  const AliasRec* __restrict__ alias;
  const uint32_t* __restrict__ gv;
  const HashEntry* __restrict__ hash;
  uint32_t* err;
  unsigned long long* steps;  // running count of produced steps (moves to a neighbour)
  unsigned long long* n2v;    // node2vec: [0] proposals drawn, [1] adjacency probes
};

__device__ __forceinline__ VertexRec load_vrec(const WalkView& W, uint32_t u) {
  const uint4 r = __ldg(reinterpret_cast<const uint4*>(W.vrec) + u);
  return VertexRec{r.x, r.y, r.z, r.w};
}

// Weighted neighbour draw at a vertex with m > 0 alias slots from aoff: slot =
// mulhi(x, m), r = mulhi64(y:z, T), group = r < thr ? own : alias, member =
// mulhi(w, cnt) (a one-member group carries its member in the slot:
// mulhi(w, 1) = 0).
struct SlotRead {
  unsigned long long thr, T, own_rc, alt_rc;
};
__device__ __forceinline__ void slot_load(SlotRead& q, const WalkView& W, uint32_t aoff, uint32_t m, const Rand4& r) {
  // The whole 32-byte slot in one 256-bit read-only load (one L1 / L2
  // request instead of two 16-byte ones; slots are 32-byte aligned and no
  // kernel writes the store while walks run).
  const AliasRec* a = W.alias + aoff + mulhi32(r.x, m);
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
      : "=l"(q.thr), "=l"(q.T), "=l"(q.own_rc), "=l"(q.alt_rc)
      : "l"(a));
}
// The drawn group: ref | count word << 32.
__device__ __forceinline__ unsigned long long slot_pick(const SlotRead& q, const Rand4& r) {
  const unsigned long long d = mulhi64(((unsigned long long)r.y << 32) | r.z, q.T);
  return d < q.thr ? q.own_rc : q.alt_rc;
}
__device__ __forceinline__ uint32_t member_load(const WalkView& W, unsigned long long rc, const Rand4& r) {
  const uint32_t ref = (uint32_t)rc, cw = (uint32_t)(rc >> 32);
  if (cw & kInlineGroup) return ref;  // one member, carried in the slot
  return __ldg(W.gv + (size_t)ref * 4 + mulhi32(r.w, cw));
}
__device__ __forceinline__ uint32_t sample_at(const WalkView& W, uint32_t aoff, uint32_t m, const Rand4& r) {
  SlotRead q;
  slot_load(q, W, aoff, m, r);
  return member_load(W, slot_pick(q, r), r);
}

// ---------------------------------------------------------------------------
// Step-at-a-time walks for the persistent kernels: a lane advances its walk
// one step per iteration and pulls a new walk as soon as its walk ends, so
// dead-ended and early-stopped walks do not idle their warp. An iteration is
// warp-converged: every lane proposes its next vertex (walk_propose), commits
// it (walk_commit), and the warp writes out finished output lines together
// (RowStage::flush).
//
// Counters: step j of walk i in job `job` draws Philox block
// (i, j, trial, job) under key seed. DeepWalk uses trial 0; PPR samples with
// trial 0 and tests its stop with trial 1; node2vec proposes with trial 2t
// and accepts with trial 2t + 1 (t = 0, 1, ...; the first step is
// first-order and takes trial 0). Row position j holds the j-th move; a walk
// that reaches a vertex without out-edges writes -1 there and pads the rest.

struct LaneWalk {
  uint32_t i;      // walk index within its job
  uint32_t j;      // step being produced
  uint32_t cur;    // current vertex
  VertexRec R;     // first-order kernels: its record, requested as soon as the vertex is known
  uint32_t lo;     // first entry of the open output line that belongs to this row
  int32_t* row;    // the walk's output row
  int32_t prev;    // previous vertex (node2vec), -1 before the first move
  uint32_t phoff;  // previous vertex's adjacency index (node2vec)
  uint32_t phmask;
  uint32_t t;       // node2vec: first trial not yet drawn of the step in progress (0 = a new step)
  uint32_t trials;  // node2vec proposals drawn by this lane (kept across its walks)
  uint32_t probes;  // node2vec adjacency-index lookups by this lane
  unsigned long long region;  // node2vec: return-region threshold of the step in progress
};

// Output lines. A lane collects its row a LINE (entries) at a time in shared
// memory; the warp then writes the line with one coalesced streaming store,
// and the end of a finished row with its -1 padding the same way. Walks are
// bound by random DRAM accesses and a row write of one 32-byte sector costs
// DRAM about as much as a read of one (R-MAT 20, 1 M walks x 80: 1138 us with
// 32-byte writes, 998 us with none): lines of 128 bytes are a quarter of the
// accesses. Lines are those of the address space, so a row may start and end
// inside one (entries before `lo` and past the row's end are not touched).
template <int LINE>
struct RowStage {
  static_assert(LINE == 8 || LINE == 16 || LINE == 32, "an entry per lane at most");
  // One lane's entries; the odd pitch spreads lanes at equal positions over the banks.
  static constexpr uint32_t kPitch = LINE + 1;

  static __device__ __forceinline__ uint32_t slot(const int32_t* p) {
    return (uint32_t)(reinterpret_cast<uintptr_t>(p) >> 2) & (LINE - 1);
  }

  // Every lane whose `out` is set writes its open line's entries [lo, last]
  // (last = slot of row position `pos`) and, when `end` (the row is
  // finished), -1 from pos + 1 to the row's end. Called by the whole warp;
  // `buf` is the warp's entries, lane l's at buf + l x kPitch.
  static __device__ __forceinline__ void flush(const int32_t* buf, bool out, bool end, LaneWalk& s, uint32_t pos,
                                               uint32_t L) {
    uint32_t todo = __ballot_sync(kFull, out);
    if (!todo) return;
    __syncwarp();  // the entries are in shared memory
    const uint32_t lane = threadIdx.x & 31;
    const int32_t* e = s.row + pos;
    const uint32_t last = slot(e);
    const unsigned long long line = reinterpret_cast<unsigned long long>(e - last);
    const uint32_t stop = end ? last + (L - pos) : last + 1;  // first entry after this write, from the line's start
    const uint32_t pack = s.lo | (last << 8);
    do {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      int32_t* const base = reinterpret_cast<int32_t*>(__shfl_sync(kFull, line, src));
      const uint32_t pk = __shfl_sync(kFull, pack, src), n = __shfl_sync(kFull, stop, src);
      const uint32_t lo = pk & 0xff, hi = pk >> 8;
      if (lane >= lo && lane < n) __stcs(base + lane, lane <= hi ? buf[src * kPitch + lane] : -1);
      for (uint32_t x = lane + 32; x < n; x += 32) __stcs(base + x, -1);
    } while (todo);
    if (out) s.lo = 0;
    __syncwarp();  // the entries may be overwritten
  }
};

// Starts walk i; returns true if it still has steps to produce. Sampling jobs
// and rows of one position complete here. `buf`: this lane's line entries.
template <int APP, int LINE, bool AHEAD = false>
__device__ __forceinline__ bool walk_begin(const WalkView& W, const WalkJobDev& J, uint32_t i, LaneWalk& s,
                                           int32_t* buf, uint32_t& moves) {
  const uint32_t start = J.starts ? J.starts[i] : J.first + i;
  const int app = APP >= 0 ? APP : J.app;
  if (app == APP_SAMPLING) {
    int32_t x = -1;
    if (start < W.n) {
      const VertexRec R = load_vrec(W, start);
      if (R.m) x = (int32_t)sample_at(W, R.aoff, R.m, philox(i, 1, 0, J.job, J.k0, J.k1));
    } else {
      set_err(W.err, E_RANGE);
    }
    J.out[i] = x;
    moves += x >= 0;
    return false;
  }
  const uint32_t L = J.L;
  if (L == 0) return false;
  s.row = J.out + (unsigned long long)i * L;
  if (start >= W.n) {
    set_err(W.err, E_RANGE);
    for (uint32_t p = 0; p < L; ++p) __stcs(s.row + p, -1);
    return false;
  }
  const bool tail = app == APP_PPR && (J.flags & kWalkPprTail);
  const uint32_t first = RowStage<LINE>::slot(s.row);
  if (first == LINE - 1 || (L == 1 && !tail)) {  // the line ends here (or the row does): nothing to collect
    __stcs(s.row, (int32_t)start);
    s.lo = 0;
    if (L == 1) {
      if (!tail) return false;
      s.lo = first;  // a tail row of one position rewrites this entry
    }
  } else {
    buf[first] = (int32_t)start;
    s.lo = first;
  }
  s.i = i;
  s.j = 1;
  s.cur = start;
  if (AHEAD) s.R = load_vrec(W, start);
  s.prev = -1;
  s.t = 0;
  return true;
}

// What a lane drew for the step in progress.
struct Proposal {
  int32_t x;             // the next vertex; -1: a dead end
  bool ok;               // node2vec: a trial was accepted (true for the other apps)
  bool stop;             // PPR: the walk ends after this move
  uint32_t hoff, hmask;  // the current vertex's adjacency index (node2vec)
};

// Draws the next vertex of a first-order walk (DeepWalk, PPR). A small launch
// is bound by the chain of a step's three reads and what lies between them, so
// little else does: the next vertex's record is requested (walk_commit) before
// the row is written and new walks are started, and the Philox blocks, which
// depend on no read, are drawn under one. DeepWalk draws `ahead`, step j + 1's
// under step j's member read (R-MAT 14, 16,384 walks x 80: 85 us with the draws
// after the record's read, 72 under it, 68 so); PPR's two blocks are longer
// than that read and stay under the record's (100,003 walks: 225 us, 227
// ahead).
//
// APP_FIRST is a table that mixes the first-order apps: its lanes draw as
// their job's app does, and read together.
template <int APP>
__device__ __forceinline__ Proposal walk_propose(const WalkView& W, const WalkJobDev& J, const LaneWalk& s,
                                                 Rand4& ahead) {
  Proposal p{-1, true, false, 0, 0};
  const bool ppr = APP == APP_PPR || (APP == APP_FIRST && J.app == APP_PPR);
  Rand4 r = ahead;
  if (ppr) {
    r = philox(s.i, s.j, 0, J.job, J.k0, J.k1);
    uint32_t ax = philox(s.i, s.j, 1, J.job, J.k0, J.k1).x;
    asm volatile("" : "+r"(r.x), "+r"(r.y), "+r"(r.z), "+r"(r.w), "+r"(ax));  // drawn before R is looked at
    p.stop = (unsigned long long)ax < J.thr_stop;
  }
  if (s.R.m) p.x = (int32_t)sample_at(W, s.R.aoff, s.R.m, r);
  if (!ppr) {
    ahead = philox(s.i, s.j + 1, 0, J.job, J.k0, J.k1);
    asm volatile("" : "+r"(p.x), "+r"(ahead.x), "+r"(ahead.y), "+r"(ahead.z), "+r"(ahead.w));  // before x is looked at
  }
  return p;
}

// node2vec steps: the warp draws trials together. A step proposes vertices
// until one is accepted; each proposal is a chain of three dependent reads,
// and how many a step takes differs from lane to lane. Which trials a step
// needs is nearly known before any read: few proposals are the previous
// vertex or its neighbours, so the first trial whose acceptance draw accepts
// any other vertex is mostly the one taken. The warp therefore lists every
// lane's trials up to that one, hands them out one per lane, 32 at a time,
// and each walk takes its lowest accepted trial (or goes on with the next
// ones): the same walk as one trial after another, with full warps of reads
// in flight and, at the end of a launch, the few walks left spread over the
// warp. First-order walks of a mixed table list their one draw, so that all
// lanes of a mixed warp read together. Bound: random DRAM reads (the
// adjacency lookups above all). R-MAT 20, 1 M walks x 40, p = 0.5, q = 2:
// 2546 us with up to three trials in turn per lane, 1933 so; 16 mixed jobs
// (1.1 M walks, up to 173 steps, q up to 4): 3986 and 1672 us.
constexpr uint32_t kTrialItems = 128;  // trials a warp lists per step
constexpr uint32_t kTrialMax = 16;     // trials a lane lists per step at most

struct TrialScratch {
  uint32_t ax[kTrialItems];    // acceptance draws, [active lane][trial]
  uint16_t item[kTrialItems];  // lane | trial << 8 | node2vec trial << 15
};

// One draw: trial t of step j of walk i at a vertex with m alias slots from
// aoff; `second`: a node2vec trial, with acceptance draw ax against the
// previous vertex and its adjacency index.
struct Trial {
  int32_t x;
  bool ok, probe;  // accepted; looked up the adjacency index
};
__device__ __forceinline__ Trial draw_trial(const WalkView& W, const WalkJobDev& V, uint32_t i, uint32_t j, uint32_t t,
                                            uint32_t aoff, uint32_t m, bool second, unsigned long long ax,
                                            int32_t prev, uint32_t phoff, uint32_t phmask) {
  Trial r{(int32_t)sample_at(W, aoff, m, philox(i, j, 2 * t, V.job, V.k0, V.k1)), true, false};
  if (second) {
    // Accepted with probability weight(class(x)) / envelope; the adjacency
    // index is read only where the class decides.
    if (r.x == prev) {
      r.ok = ax < V.thr_ret;
    } else if (ax >= (V.thr_in < V.thr_out ? V.thr_in : V.thr_out)) {
      r.probe = true;
      r.ok = ax < (hash_has(W.hash + phoff, phmask, (uint32_t)r.x) ? V.thr_in : V.thr_out);
    }
    r.ok = r.ok || t + 1 == kMaxNode2vecTrials;
  }
  return r;
}

// One step of every active lane's walk; `jobs` is the job table (jid indexes
// it) or the one job.
template <int APP>
__device__ __forceinline__ Proposal warp_propose(const WalkView& W, const WalkJobDev* __restrict__ jobs, uint32_t jid,
                                                 LaneWalk& s, bool active, TrialScratch& sc) {
  const uint32_t lane = threadIdx.x & 31;
  const WalkJobDev& J = jobs[jid];
  const int app = APP >= 0 ? APP : J.app;
  VertexRec R{0, 0, 0, 0};
  if (active) R = load_vrec(W, s.cur);
  const bool n2v = active && app == APP_NODE2VEC && s.prev >= 0;
  // Trials listed per lane: all lanes' lists fit the scratch.
  const uint32_t am = __ballot_sync(kFull, active), na = __popc(am);
  const uint32_t cap = min(kTrialMax, na > 16 ? kTrialItems / 32 : kTrialItems >> (32 - __clz((na - 1) | 1)));
  const uint32_t mine = __popc(am & lanemask_lt()) * cap;  // this lane's acceptance draws in the scratch
  Proposal p{-1, true, false, 0, 0};
  uint32_t n = active ? 1u : 0u;  // trials listed
  if (n2v || (active && app == APP_PPR)) {
    n = 0;
    bool more;
    do {
      const uint32_t ax = philox(s.i, s.j, 2 * (s.t + n) + 1, J.job, J.k0, J.k1).x;
      more = false;
      if (APP < 0 && app == APP_PPR) {
        p.stop = (unsigned long long)ax < J.thr_stop;
      } else {
        sc.ax[mine + n] = ax;
        more = ax >= J.thr_out && n + 1 < cap && s.t + n + 1 < kMaxNode2vecTrials;
      }
      ++n;
    } while (more);
  }
  p.hoff = R.hoff, p.hmask = R.hmask;
  if (!R.m) n = 0;
  // A new step's return-region lookup (below) starts here, beside the trials.
  const bool ret = n2v && R.m && s.t == 0 && J.ret_excess > 0.0;
  HashPeek rp;
  if (ret) hash_peek(rp, W.hash + R.hoff, R.hmask, (uint32_t)s.prev);
  constexpr uint32_t kNone = 0xffffffffu;
  uint32_t won = kNone, probed = 0;  // the accepted trial; this lane's trials that looked up the adjacency index
  if (!__any_sync(kFull, n > 1)) {
    // A draw per lane at most (DeepWalk, PPR, q <= 1): each draws its own.
    // R-MAT 16, p = q = 1, 4,000 walks x 80: 143 us listed, 114 so; p = q =
    // 0.25: 257 and 220. (Walks with q > 1 seldom get here: 1 M walks x 40 on
    // R-MAT 20 take 1952 us without this and 1958 with it.)
    if (n) {
      const Trial r = draw_trial(W, J, s.i, s.j, s.t, R.aoff, R.m, n2v, n2v ? sc.ax[mine] : 0u, s.prev, s.phoff, s.phmask);
      if (r.ok) won = 0, p.x = r.x;
      probed = r.probe;
    }
  } else {
    const uint32_t incl = warp_incl_scan(n, lane), off = incl - n;
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    for (uint32_t k = 0; k < n; ++k) sc.item[off + k] = (uint16_t)(lane | k << 8 | (n2v ? 1u << 15 : 0u));
    __syncwarp();
    for (uint32_t base = 0; base < total; base += 32) {
      const bool valid = base + lane < total;
      const uint32_t it = valid ? sc.item[base + lane] : 0u;
      const int src = it & 31;
      const uint32_t k = (it >> 8) & 0x7f;
      const uint32_t vi = __shfl_sync(kFull, s.i, src), vj = __shfl_sync(kFull, s.j, src);
      const uint32_t vt = __shfl_sync(kFull, s.t, src) + k;
      const uint32_t vaoff = __shfl_sync(kFull, R.aoff, src), vm = __shfl_sync(kFull, R.m, src);
      const int32_t vprev = __shfl_sync(kFull, s.prev, src);
      const uint32_t vphoff = __shfl_sync(kFull, s.phoff, src), vphmask = __shfl_sync(kFull, s.phmask, src);
      const WalkJobDev& V = jobs[__shfl_sync(kFull, jid, src)];
      Trial r{-1, false, false};
      if (valid) {
        const uint32_t ax = sc.ax[__popc(am & ((1u << src) - 1u)) * cap + k];
        r = draw_trial(W, V, vi, vj, vt, vaoff, vm, it >> 15, ax, vprev, vphoff, vphmask);
      }
      const uint32_t oks = __ballot_sync(kFull, r.ok), probes = __ballot_sync(kFull, r.probe);
      const uint32_t lo = max(off, base), hi = min(off + n, base + 32);
      int from = 0;
      bool take = false;
      if (lo < hi && won == kNone) {  // this lane's trials among the 32
        const uint32_t here = kFull >> (32 - (hi - lo)), first = lo - base;
        const uint32_t acc = (oks >> first) & here;
        probed |= ((probes >> first) & here) << (lo - off);
        if (acc) {
          from = (int)(first + __ffs(acc) - 1);
          won = base + from - off;
          take = true;
        }
      }
      const int32_t x = __shfl_sync(kFull, r.x, from);
      if (take) p.x = x;
    }
  }
  if (n2v && R.m) {
    // Return region: when 1/p exceeds the envelope max(1, 1/q), the excess
    // mass (ret_excess x w(cur -> prev)) returns to prev directly, with
    // probability D / (T + D) per trial (word y of the acceptance block): the
    // first trial in the region ends the step unless an earlier one did.
    if (s.t == 0) {
      s.region = 0;
      if (ret) {
        const int e = hash_settle(rp, W.hash + R.hoff, R.hmask, (uint32_t)s.prev);
        ++s.probes;
        if (e >= 0 && __ldg(&W.hash[R.hoff + e].cnt) > 0) {
          const unsigned long long wp = __ldg(&W.hash[R.hoff + e].wsum);
          const double T = (double)__ldg(&W.alias[R.aoff].T);
          const double D = __dmul_rn(J.ret_excess, (double)wp);
          s.region = prob_threshold_dev(__ddiv_rn(D, __dadd_rn(T, D)));
        }
      }
    }
    uint32_t drawn = won == kNone ? n : won + 1;  // trials up to the accepted one
    p.ok = won != kNone;
    if (s.region) {
      const uint32_t upto = drawn;
      for (uint32_t k = 0; k < upto; ++k)
        if ((unsigned long long)philox(s.i, s.j, 2 * (s.t + k) + 1, J.job, J.k0, J.k1).y < s.region) {
          p.x = s.prev;
          p.ok = true;
          drawn = k;
          break;
        }
    }
    s.trials += drawn;
    s.probes += __popc(probed & ((1u << drawn) - 1u));
    if (!p.ok) s.t += n;
  }
  __syncwarp();  // the scratch is free for the next step
  return p;
}

// Takes the proposal as the walk's next move. Returns false when the walk has
// ended; `out` is set when the row's open line must be written (RowStage::
// flush up to row position `pos`).
template <int APP, int LINE, bool AHEAD = false>
__device__ __forceinline__ bool walk_commit(const WalkView& W, const WalkJobDev& J, LaneWalk& s, const Proposal& p, int32_t* buf,
                                            uint32_t& moves, bool& out, uint32_t& pos) {
  const int app = APP >= 0 ? APP : J.app;
  const bool tail = app == APP_PPR && (J.flags & kWalkPprTail);
  const uint32_t L = J.L;
  pos = s.j < L ? s.j : L - 1;
  const uint32_t at = RowStage<LINE>::slot(s.row + pos);
  bool done = p.x < 0;
  buf[at] = p.x;
  if (!done) {
    ++moves;
    if (app == APP_NODE2VEC) {
      s.prev = (int32_t)s.cur;
      s.phoff = p.hoff;
      s.phmask = p.hmask;
      s.t = 0;
    }
    s.cur = (uint32_t)p.x;
    ++s.j;
    done = p.stop || (s.j >= L && !tail) || (tail && s.j >= kMaxPprSteps);
    if (AHEAD && !done) s.R = load_vrec(W, s.cur);
  }
  // A tail walk rewrites its last position until it stops.
  out = done || (at == LINE - 1 && !(tail && pos == L - 1));
  return !done;
}

// One atomic per warp: adds the warp's produced steps to the running count.
__device__ __forceinline__ void add_steps(const WalkView& W, unsigned long long mine) {
#pragma unroll
  for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(W.steps, mine);
}

// The same for the node2vec proposal and probe counts (zero, and folded
// away, in kernels without node2vec walks).
__device__ __forceinline__ void add_n2v(const WalkView& W, const LaneWalk& s) {
  unsigned long long t = s.trials, p = s.probes;
#pragma unroll
  for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(kFull, t, o), p += __shfl_xor_sync(kFull, p, o);
  if ((threadIdx.x & 31) == 0 && (t | p)) atomicAdd(W.n2v, t), atomicAdd(W.n2v + 1, p);
}

}  // namespace bingo
