// The host side of nsp_b200/csrc/runrules.h, for tests/test_run_rules_cpu.py.
#include "runrules.h"

#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

using namespace nspb;

extern "C" {

int max_a(void) { return kRunMaxA; }
int max_ip(void) { return kRunMaxIp; }

// Products of a row as the kernels add them: 32 lengths at a time in 32 bits, and
// no further once there are too many.
int row_products(const int *len, int na) {
  int total = 0;
  for (int c = 0; c < na; c += 32) {
    unsigned sum = 0;
    for (int t = c; t < na && t < c + 32; ++t) sum += (unsigned)run_len(len[t]);
    total += (int)sum;
    if (total > kRunMaxIp) return kRunMaxIp + 1;
  }
  return total;
}

// Values of a tile's one segment of B as the kernel counts them (32 bits), or -1
// where its rows may not share a tile.
int tile_values(int step, int rows, int len) {
  if (!run_step_fits(step, rows)) return -1;
  return (int)((unsigned)(rows - 1) * (unsigned)step + (unsigned)len);
}

// Warps of a block decide whether to give up while the flag is raised between
// the views of warp `after` and of the next one. Returns how many of them stop.
int warps_that_stop(int warps, int after) {
  std::mutex m;
  std::condition_variable cv;
  int turn = 0, here = 0, stops = 0;
  bool lost = false, vote = false;
  std::vector<std::thread> block;
  for (int w = 0; w < warps; ++w)
    block.emplace_back([&, w] {
      auto view = [&] {  // in turn, so that the flag changes where it should
        std::unique_lock<std::mutex> l(m);
        cv.wait(l, [&] { return turn == w; });
        const bool seen = lost;
        if (w == after) lost = true;
        ++turn;
        cv.notify_all();
        return seen;
      };
      auto any = [&](bool yes) {  // a barrier that votes
        std::unique_lock<std::mutex> l(m);
        vote = vote || yes;
        ++here;
        cv.notify_all();
        cv.wait(l, [&] { return here == warps; });
        return vote;
      };
      const bool stop = run_gives_up(view, any);
      std::lock_guard<std::mutex> l(m);
      stops += stop;
    });
  for (auto &t : block) t.join();
  return stops;
}
}
