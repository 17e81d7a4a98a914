// barrier_check.cc -- the grid barrier's counter arithmetic
// (rdmce_b200/csrc/barrier.h) past 2^32 arrivals.  Built and run by
// tests/test_grid_barrier.py.
//
//   barrier_check <blocks> <first count> <barriers>
//
// Blocks arrive in a scrambled order; each polls after every arrival, the way
// k_peel_rounds does.  Fails when a block passes before the last one arrived,
// or has not passed after it.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "barrier.h"

int main(int argc, char **argv) {
  if (argc != 4) return 2;
  const uint32_t blocks = (uint32_t)std::strtoul(argv[1], nullptr, 0);
  const uint32_t first = (uint32_t)std::strtoul(argv[2], nullptr, 0);
  const int barriers = std::atoi(argv[3]);
  uint32_t arrived = first, target = first;
  uint64_t rng = 1;
  for (int b = 0; b < barriers; b++) {
    target += blocks;
    std::vector<bool> in(blocks, false);
    for (uint32_t k = 0; k < blocks; k++) {
      rng = rng * 6364136223846793005ULL + 1442695040888963407ULL;
      uint32_t x = (uint32_t)(rng >> 33) % blocks;
      while (in[x]) x = (x + 1) % blocks;
      in[x] = true;
      arrived++;
      const bool last = k + 1 == blocks;
      if (mce::barrier_reached(arrived, target) != last) {
        std::fprintf(stderr, "barrier %d: %s after %u of %u arrivals (count %u, target %u)\n", b,
                     last ? "not passed" : "passed", k + 1, blocks, arrived, target);
        return 1;
      }
    }
    // a quick block may have arrived at the next barrier when a slow one polls
    for (uint32_t ahead = 1; ahead < blocks; ahead++)
      if (!mce::barrier_reached(arrived + ahead, target)) {
        std::fprintf(stderr, "barrier %d: a slow block waits on (count %u, target %u)\n", b, arrived + ahead, target);
        return 1;
      }
  }
  std::puts("BARRIER OK");
  return 0;
}
