// CPU-thread model of a loop of levels with one barrier a level (the one-CTA
// BFS): host threads run its words' turns with the same code as the kernel
// (wgm_protocol.h).  Built and driven by tests/test_levels_model.py; test
// code only.
//
// A planted mistake lives here, never in the product: with `planted` the
// first thread clears the flag of the level just ended, which the others may
// still have to read.
#include <atomic>
#include <barrier>
#include <chrono>
#include <thread>
#include <vector>

#include "../../include/wgm_protocol.h"

// `threads` run `levels` levels, every one of which raises its flag and hands
// one unit of work to the next.  Thread 0 never waits; the last one reads a
// level's flag only when thread 0 has cleared its words at the top of the next
// (or after a while, at the end).  out[0]: threads that took a level for
// the last one too soon, out[1]: sizes that were not 1 at the top of a level.
extern "C" int model_levels(int planted, int threads, int levels, int *out) {
  std::atomic<int> size[3] = {0, 1, 0}, flag[3] = {0, 0, 0};
  std::atomic<int> top{0}, early{0}, wrong{0};
  std::barrier<> bar(threads);
  std::vector<std::thread> th;
  for (int t = 0; t < threads; t++)
    th.emplace_back([&, t] {
      wgm_proto_levels w{1, 2, 0};
      for (int L = 1; L <= levels; L++) {
        if (size[w.now].load() != 1) wrong++;
        if (t == 0) {
          size[w.size_to_clear()].store(0);
          flag[planted ? w.last : w.flag_to_clear()].store(0);
          top.store(L);
        }
        flag[w.now].store(1);
        if (t == threads - 1) size[w.next].fetch_add(1);
        bar.arrive_and_wait();
        if (t == threads - 1) {
          const auto t0 = std::chrono::steady_clock::now();
          while (top.load() <= L &&
                 std::chrono::steady_clock::now() - t0 < std::chrono::milliseconds(20)) {
          }
        }
        if (!flag[w.now].load()) {
          early++;
          bar.arrive_and_drop();
          return;
        }
        w.step();
      }
    });
  for (auto &t : th) t.join();
  out[0] = early.load();
  out[1] = wrong.load();
  return 0;
}
