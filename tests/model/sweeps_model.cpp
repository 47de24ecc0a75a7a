// CPU model of the sweeps that settle a colour block's inner edges: every edge is
// a thread that reads its source, reads its target and stores source + 1 over a
// target that is not larger, three looks a sweep, in any interleaving of those steps.
// Its bound is the kernel's (wgm_protocol.h).  Built and driven by
// tests/test_sweeps_model.py; test code only.
#include <cstdint>
#include <random>
#include <vector>

#include "../../include/wgm_protocol.h"

// Edges src[e] -> dst[e] over the words col[].  stall 0: steps in random order;
// 1: of the edges into a target, the one of the smallest source reads first and
// stores last.  Returns the sweeps run, the clean one included, or -1 when the bound
// did not do.
extern "C" int model_sweeps(int edges, const int *src, const int *dst, int *col, int stall,
                            uint64_t seed) {
  std::mt19937_64 rng(seed);
  const int bound = wgm_proto_chain_sweeps(edges);
  for (int sweep = 1; sweep <= bound; sweep++) {
    bool changed = false;
    std::vector<int> step(edges, 0), c(edges), d(edges), live;
    for (int e = 0; e < edges; e++) live.push_back(e);
    while (!live.empty()) {
      size_t at = rng() % live.size();
      if (stall) {  // reads first, then stores by falling source
        size_t best = 0;
        long best_key = -1;
        for (size_t k = 0; k < live.size(); k++) {
          const int e = live[k];
          const long key = step[e] < 2 ? (1L << 40) - step[e] : c[e];
          if (key > best_key) best_key = key, best = k;
        }
        at = best;
      }
      const int e = live[at];
      switch (step[e] % 3) {
        case 0: c[e] = col[src[e]]; break;
        case 1: d[e] = col[dst[e]]; break;
        case 2:
          if (c[e] >= d[e]) {
            col[dst[e]] = c[e] + 1;
            changed = true;
          }
      }
      if (++step[e] == 9) {
        live[at] = live.back();
        live.pop_back();
      }
    }
    if (!changed) return sweep;
  }
  return -1;
}
