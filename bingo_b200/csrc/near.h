// Which of an edge's back-pointers are brought near ahead of its removal
// (plain C++, host and device).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define BINGO_NEAR_HD __host__ __device__ __forceinline__
#else
#define BINGO_NEAR_HD inline
#endif

namespace bingo {

// An edge's run has one back-pointer per set bit of its weight w; the first
// one is requested, and with it the one this many entries on (at most eight
// entries: one 32-byte sector, or the two that hold them), never past the run:
// the pool may end there. A deleted edge (w = 0) has none.
BINGO_NEAR_HD uint32_t near_last(uint32_t w) {
#ifdef __CUDA_ARCH__
  const uint32_t run = __popc(w);
#else
  const uint32_t run = __builtin_popcount(w);
#endif
  return run > 8 ? 7u : run ? run - 1 : 0u;
}

}  // namespace bingo
