// Autotuner: picks the launch and batching knobs (Tuning) by timing the
// caller's own sample workload on the live graph.
//
// Walk knobs are timed on the job set through the batched walk path; walks
// do not change the graph, and no knob changes any walk, so the outputs are
// simply rewritten. Update knobs are timed by applying the sample batch and
// then restoring the store from a device copy taken before the first trial,
// so the graph is the same when the call returns.
//
// Search: tune_search.h.
#include <algorithm>
#include <chrono>

#include "engine.cuh"

namespace bingo {

void Engine::autotune(const bingo_tune_request& R, bingo_tune_report* out) {
  const NvtxRange nvtx_("bingo autotune");
  require_loaded();
  require_idle();
  if (!R.n_jobs && !R.n_ins && !R.n_del) throw Error(BINGO_ERR_INVALID_ARGUMENT, "empty tuning request");
  if (R.n_jobs && !R.jobs) throw Error(BINGO_ERR_INVALID_ARGUMENT, "null job array");
  const int reps = R.repeats ? (int)std::min<uint32_t>(R.repeats, 64) : 3;
  const Tuning start = tuning_;
  Tuning best = tuning_;
  uint32_t cand = 0;

  auto wall_ms = [&](auto&& fn) {
    cuda_check(cudaStreamSynchronize(stream_), "tune");
    const auto t0 = std::chrono::steady_clock::now();
    fn();
    const int st = sync();
    if (st) throw Error(st, last_error);
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  };

  double walk_start = -1, walk_best = -1;
  if (R.n_jobs) {
    auto once = [&](const Tuning& t) {
      tuning_ = t;
      return wall_ms([&] { walk(R.jobs, R.n_jobs, BINGO_WALK_BATCHED); });
    };
    try {
      KnobSearch<decltype(once)> s(best, reps, once);
      bool mixed = false;
      for (uint32_t j = 1; j < R.n_jobs; ++j) mixed |= R.jobs[j].app != R.jobs[0].app;
      search_walk_knobs(s, R.n_jobs > 1, mixed);
      best = s.best, walk_start = s.ms_start, walk_best = s.ms_best, cand += s.candidates;
    } catch (...) {
      tuning_ = start;
      throw;
    }
  }

  double upd_start = -1, upd_best = -1;
  if (R.n_ins || R.n_del) {
    if ((R.n_ins && (!R.ins_src || !R.ins_dst || !R.ins_w)) || (R.n_del && (!R.del_u || !R.del_slot)))
      throw Error(BINGO_ERR_INVALID_ARGUMENT, "null update array");
    StateCopy snap;
    if (save_state(snap)) {
      auto once = [&](const Tuning& t) {
        tuning_ = t;
        restore_state(snap);
        return wall_ms([&] {
          if (R.n_ins) insert(R.ins_src, R.ins_dst, R.ins_w, R.n_ins, nullptr);
          if (R.n_del) erase(R.del_u, R.del_slot, R.n_del);
        });
      };
      try {
        KnobSearch<decltype(once)> s(best, reps, once);
        search_update_knobs(s, std::max(R.n_ins, R.n_del));
        best = s.best, upd_start = s.ms_start, upd_best = s.ms_best, cand += s.candidates;
        restore_state(snap);
      } catch (...) {
        tuning_ = start;
        try {
          restore_state(snap);
        } catch (...) {
        }
        snap.release();
        throw;
      }
      snap.release();
    }
  }

  tuning_ = best;
  if (out) {
    *out = bingo_tune_report{};
    out->best.walk_chunk = best.walk_chunk;
    out->best.walk_blocks_per_sm = best.walk_blocks_per_sm;
    out->best.walk_split = best.walk_split;
    out->best.walk_order = best.walk_order;
    out->best.update_chunk = best.update_chunk;
    out->best.apply_blocks_per_sm = best.apply_blocks_per_sm;
    out->walk_ms_start = walk_start;
    out->walk_ms_best = walk_best;
    out->update_ms_start = upd_start;
    out->update_ms_best = upd_best;
    out->candidates = cand;
  }
}

}  // namespace bingo
