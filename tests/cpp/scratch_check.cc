// scratch_check.cc -- range solves when the vertex pass's lists cannot be
// allocated.  Built and run by tests/test_gpu_calls_kept.py.
//
//   scratch_check <pairs file> <number of pairs>
//
// The file holds the pairs' first and then their second labels, 32 bits each.
// A full solve and two cut ranges go once with the lists and once with the
// default scratch turning the larger buffer down; results and root counts have
// to agree, and the second time there is one enumeration launch a solve.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "rdmce.h"
#include "scratch.h"

#define CHECK(cond)                                                           \
  do {                                                                        \
    if (!(cond)) {                                                            \
      std::fprintf(stderr, "check failed at line %d: %s\n", __LINE__, #cond); \
      return 1;                                                               \
    }                                                                         \
  } while (0)

int main(int argc, char **argv) {
  if (argc != 3) return 2;
  const size_t pairs = std::strtoull(argv[2], nullptr, 10);
  std::vector<uint32_t> uv(2 * pairs);
  std::FILE *f = std::fopen(argv[1], "rb");
  CHECK(f && std::fread(uv.data(), 4, uv.size(), f) == uv.size());
  std::fclose(f);
  mce_options o;
  mce_default_options(&o);
  o.spin_limit = 1 << 22;
  mce_graph *g = nullptr;
  CHECK(mce_graph_from_coo(uv.data(), uv.data() + pairs, pairs, &o, &g) == MCE_OK);
  mce_graph_info info;
  CHECK(mce_graph_info_get(g, &info) == MCE_OK);
  const uint64_t m = info.num_edges, cut[4] = {0, m / 3 + 1, m / 2 + 1, m};
  static mce_result with, without;
  for (int part = -1; part < 3; part++) {
    o.root_begin = part < 0 ? 0 : cut[part];
    o.root_end = part < 0 ? m : cut[part + 1];
    const uint64_t roots = o.root_end - o.root_begin;
    mce::Scratch *scr = mce::default_scratch(0);
    scr->most[3] = 0;
    CHECK(mce_solve(g, &o, &with) == MCE_OK);
    CHECK(with.launches == 3 && with.roots == roots);
    scr->release();
    scr->most[3] = roots * 4;
    CHECK(mce_solve(g, &o, &without) == MCE_OK);
    CHECK(without.launches == 1 && without.roots == roots);
    CHECK(with.count == without.count && with.checksum == without.checksum && with.max_size == without.max_size);
    for (int i = 0; i < MCE_HIST_LEN; i++) CHECK(with.hist[i] == without.hist[i]);
    if (part < 0) std::printf("SCRATCH OK count %llu checksum %llu\n", (unsigned long long)with.count,
                              (unsigned long long)with.checksum);
    scr->most[3] = roots * 4 - 4;  // not even the deferred roots' list
    scr->release();
    CHECK(mce_solve(g, &o, &without) == MCE_ERR_OUT_OF_MEMORY);
  }
  mce::default_scratch(0)->most[3] = 0;
  CHECK(mce_solve(g, &o, &with) == MCE_OK);
  mce_graph_free(g);
  return 0;
}
