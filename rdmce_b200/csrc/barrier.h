// barrier.h -- arithmetic of the grid barrier (preprocess.cu), also built into
// a host test.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MCE_HD __host__ __device__
#else
#define MCE_HD
#endif

namespace mce {

// A barrier counts arrivals in 32 bits and is never reset; `target` is the
// count at which this barrier is complete.  A block is at most one barrier
// ahead of another, so the count is within a grid of the target on either side
// and their difference modulo 2^32 has the right sign.  Comparing the values
// themselves fails after 2^32 / 148 = 2.9e7 barriers: a path of 5.8e7 vertices
// peels in that many rounds.
MCE_HD constexpr bool barrier_reached(uint32_t seen, uint32_t target) { return (int32_t)(seen - target) >= 0; }

// Counts start shortly before the wrap, so that every grid peel passes it.
constexpr uint32_t kBarrierStart = 0u - 1000u;

}  // namespace mce
