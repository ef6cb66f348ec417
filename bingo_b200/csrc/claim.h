// Work counters of the persistent walk kernels and the arithmetic of handing
// walks out, for totals up to 2^32 - 1 (plain C++, host and device).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define BINGO_HD __host__ __device__ __forceinline__
#else
#define BINGO_HD inline
#endif

namespace bingo {

// One launch's work counter: zero at launch, zeroed again by its last warp.
// `next` is 64 bits wide because every warp adds to it once more after the
// last walk: in 32 bits a total near 2^32 would wrap and be handed out again.
struct WalkQueue {
  unsigned long long next;  // next unclaimed walk
  uint32_t done;            // warps that have finished
  uint32_t pad;
};

constexpr uint32_t kClaimMin = 4, kClaimMax = 32;

// The claim that started at counter value `base`: walks [*begin, *end), or
// none (false) when all `total` are claimed.
BINGO_HD bool claim_range(unsigned long long base, uint32_t total, uint32_t chunk, uint32_t* begin, uint32_t* end) {
  if (base >= total) return false;
  *begin = (uint32_t)base;
  const uint32_t left = total - *begin;
  *end = *begin + (chunk < left ? chunk : left);
  return true;
}

// Size of a warp's next claim in tables of several apps, from its last one and
// the steps that one lasted (the first fill of its lanes: kClaimMin each).
// What a warp holds unstarted waits for its lanes, which is worst for long
// walks; but short ones (PPR) use four up in less than a step, and the warp
// then waits for the counter at every step. A claim that lasted up to 4 steps
// is doubled, one that lasted 16 or more halved. R-MAT 22, sixteen tables of 16
// jobs: the one with most short walks 12.87 ms at 4 walks per claim, 11.96 at
// 32, 12.38 so; one of long walks 2.20, 3.19 and 2.18; all of them 120.3, 124.3
// and 119.3. (Lines at 8 and 24, and at 12 and 48, within 0.2 % of these.)
BINGO_HD uint32_t next_claim(uint32_t last, uint32_t steps) {
  if (steps <= 4) return last < kClaimMax ? last * 2 : kClaimMax;
  if (steps >= 16) return last > kClaimMin ? last / 2 : kClaimMin;
  return last;
}

// Each of `warps` warps' share of `total` items, rounded up (without
// total + warps - 1, which does not fit 32 bits for the largest totals).
BINGO_HD uint32_t walk_share(uint32_t total, uint32_t warps) {
  return total / warps + (total % warps != 0 ? 1u : 0u);
}

}  // namespace bingo
