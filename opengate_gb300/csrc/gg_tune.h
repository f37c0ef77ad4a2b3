// gg_tune.h - the search of gg_batch_autotune.  Plain C++, so that it is tested with made-up times.
#pragma once

#include <algorithm>
#include <cstdint>

namespace gg {

// What a batched run's launches depend on: resident blocks per SM (of 256 threads, as
// in gg_device_opts), histories a warp claims, histories per batch.
struct TunePoint {
  int blocks, chunk;
  int64_t batch;
};

struct TuneSearch {
  TunePoint best;
  int points = 0;                    // configurations timed
  double start_ms = 0, best_ms[3]{}; // of the start (median), of the best (median, least, most)
};

// Times the start, then every launch shape of the pooled kernel (block: its full
// block's threads) x claim chunk x batch length (all `total` histories in one
// generate / transport / flush sequence, or in 2 or 4); the phase thresholds of the
// options do not exist in that kernel.  The start stays the best unless a point is
// faster; its blocks are given as the full block's when they are not set, which is
// the same launch.  time_point(point, ms[3]): 0 or a status that ends the search.
template <typename Time>
int tune_search(TunePoint start, int block, uint64_t total, Time &&time_point, TuneSearch &r) {
  const int full = (block + 255) / 256;
  start.blocks = start.blocks <= 0 ? full : std::min(std::max(start.blocks, 2), std::max(full, 2));
  r = TuneSearch{};
  r.best = start;
  int st = time_point(start, r.best_ms);
  if (st) return st;
  r.points = 1;
  r.start_ms = r.best_ms[0];
  for (int blocks = std::min(2, full); blocks <= full; ++blocks)
    for (int chunk : {64, 256, 1024})
      for (int parts : {1, 2, 4}) {
        const TunePoint p{blocks, chunk, std::max<int64_t>(1, (int64_t)((total + parts - 1) / parts))};
        double t[3];
        if ((st = time_point(p, t))) return st;
        ++r.points;
        if (t[0] < r.best_ms[0]) {
          std::copy(t, t + 3, r.best_ms);
          r.best = p;
        }
      }
  return 0;
}

}  // namespace gg
