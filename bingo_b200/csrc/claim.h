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

// The claim that started at counter value `base`: walks [*begin, *end), or
// none (false) when all `total` are claimed.
BINGO_HD bool claim_range(unsigned long long base, uint32_t total, uint32_t chunk, uint32_t* begin, uint32_t* end) {
  if (base >= total) return false;
  *begin = (uint32_t)base;
  const uint32_t left = total - *begin;
  *end = *begin + (chunk < left ? chunk : left);
  return true;
}

// Each of `warps` warps' share of `total` items, rounded up (without
// total + warps - 1, which does not fit 32 bits for the largest totals).
BINGO_HD uint32_t walk_share(uint32_t total, uint32_t warps) {
  return total / warps + (total % warps != 0 ? 1u : 0u);
}

}  // namespace bingo
