// The autotuner's search over the launch and batching knobs, apart from what
// it times (plain C++).
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace bingo {

// Launch and batching knobs (bingo_tuning); none changes any result.
struct Tuning {
  uint32_t walk_chunk = 0;          // 0 = each walk kernel's default (walk_default_chunk)
  uint32_t walk_blocks_per_sm = 0;  // 0 = each walk kernel's default (walk_default_bps)
  uint32_t walk_split = 0;
  uint32_t walk_order = 1;
  uint32_t update_chunk = 0;  // 0 = whole batch
  uint32_t apply_blocks_per_sm = 8;
};

// One search: `once(t)` runs the sample under knobs t and returns its time. A
// candidate replaces the current choice only when its median is at least 1 %
// lower, so noise does not move the knobs; each knob still comes from the
// lowest of several noisy medians, so the choice is timed against the knobs
// the search started from once more, the two in turn, and has to win again.
template <class Once>
class KnobSearch {
 public:
  KnobSearch(const Tuning& start, int reps, Once once)
      : best(start), start_(start), reps_(reps), once_(once), ms_start(-1), ms_best(-1) {
    ms_start = ms_best = time(start);
  }

  void try_knob(uint32_t Tuning::*f, const std::vector<uint32_t>& values) {
    for (uint32_t x : values) {
      if (best.*f == x) continue;
      Tuning t = best;
      t.*f = x;
      const double ms = time(t);
      if (ms < ms_best * 0.99) ms_best = ms, best = t;
    }
  }

  void confirm() {
    if (same(best, start_)) return;
    std::vector<double> a, b;
    for (int r = 0; r <= reps_; ++r) {
      const double x = once_(start_), y = once_(best);
      if (r) a.push_back(x), b.push_back(y);
    }
    ms_start = median(a), ms_best = median(b);
    if (!(ms_best < ms_start * 0.99)) best = start_, ms_best = ms_start;
  }

  Tuning best;

 private:
  const Tuning start_;
  const int reps_;
  Once once_;

  static bool same(const Tuning& x, const Tuning& y) {
    return x.walk_chunk == y.walk_chunk && x.walk_blocks_per_sm == y.walk_blocks_per_sm &&
           x.walk_split == y.walk_split && x.walk_order == y.walk_order && x.update_chunk == y.update_chunk &&
           x.apply_blocks_per_sm == y.apply_blocks_per_sm;
  }

  static double median(std::vector<double> v) {
    std::sort(v.begin(), v.end());
    const size_t m = v.size() / 2;
    return v.size() % 2 ? v[m] : 0.5 * (v[m - 1] + v[m]);
  }

  double time(const Tuning& t) {
    std::vector<double> v;
    for (int r = 0; r <= reps_; ++r) {
      const double ms = once_(t);
      if (r) v.push_back(ms);  // the first run warms up
    }
    ++candidates;
    return median(v);
  }

 public:
  double ms_start, ms_best;
  uint32_t candidates = 0;
};

// Walk knobs of a sample of jobs, in a fixed order: walk_chunk, walk_split,
// walk_order, walk_blocks_per_sm, a second look at walk_chunk around the pick.
// The list holds every kernel's default (0, and the 4 and 8 it stands for).
template <class Search>
void search_walk_knobs(Search& s, bool several_jobs, bool several_apps) {
  s.try_knob(&Tuning::walk_chunk, {0, 2, 4, 8, 16, 32, 64, 128, 256});
  if (several_apps) s.try_knob(&Tuning::walk_split, {0, 1});
  if (several_jobs) s.try_knob(&Tuning::walk_order, {1, 0});
  s.try_knob(&Tuning::walk_blocks_per_sm, {0, 6, 4, 3, 2});
  std::vector<uint32_t> around;  // 0 (each kernel's default) has no neighbours
  if (s.best.walk_chunk > 1) around.push_back(s.best.walk_chunk / 2);
  if (s.best.walk_chunk && s.best.walk_chunk < 1024) around.push_back(s.best.walk_chunk * 2);
  s.try_knob(&Tuning::walk_chunk, around);
  s.confirm();
}

// Update knobs of a sample whose larger batch has kmax edges.
template <class Search>
void search_update_knobs(Search& s, uint64_t kmax) {
  std::vector<uint32_t> chunks{0};
  for (uint64_t c = kmax / 2; c >= 16384 && chunks.size() < 4; c /= 2) chunks.push_back((uint32_t)c);
  s.try_knob(&Tuning::update_chunk, chunks);
  s.try_knob(&Tuning::apply_blocks_per_sm, {8, 4, 16, 32});
  s.confirm();
}

}  // namespace bingo
