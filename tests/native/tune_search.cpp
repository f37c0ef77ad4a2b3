// The batch autotuner's search with made-up times.
#include <cstdio>
#include <set>
#include <tuple>

#include "../../opengate_gb300/csrc/gg_tune.h"

#define REQUIRE(x)                            \
  if (!(x)) {                                 \
    std::printf("line %d: %s\n", __LINE__, #x); \
    return 1;                                 \
  }

int main() {
  using gg::TunePoint;
  const TunePoint start{0, 64, (int64_t)1 << 26};
  const uint64_t total = 1000003;
  // nothing beats the start, by however little: it stays, as the launch it was (no set count: the full block)
  for (double slower : {0.0, 0.001, 5.0}) {
    int calls = 0;
    gg::TuneSearch r;
    std::set<std::tuple<int, int, int64_t>> points;
    const int st = gg::tune_search(start, 640, total, [&](const TunePoint &p, double t[3]) {
      points.insert({p.blocks, p.chunk, p.batch});
      t[0] = t[1] = t[2] = calls++ == 0 ? 10.0 : 10.0 + slower;
      return 0;
    }, r);
    REQUIRE(st == 0 && r.points == calls && calls == 19 && points.size() == 19);  // no point twice
    REQUIRE(r.best.blocks == 3 && r.best.chunk == 64 && r.best.batch == start.batch);
    REQUIRE(r.best_ms[0] == 10.0 && r.start_ms == 10.0);
  }
  // the fastest of several faster points, with its times
  {
    gg::TuneSearch r;
    REQUIRE(gg::tune_search(start, 640, total, [&](const TunePoint &p, double t[3]) {
      t[0] = p.blocks == 2 && p.chunk == 256 && p.batch == 500002 ? 7.0 : (p.chunk == 1024 ? 8.0 : 9.0);
      t[1] = t[0] - 1;
      t[2] = t[0] + 1;
      return 0;
    }, r) == 0);
    REQUIRE(r.best.blocks == 2 && r.best.chunk == 256 && r.best.batch == 500002);
    REQUIRE(r.best_ms[0] == 7.0 && r.best_ms[1] == 6.0 && r.best_ms[2] == 8.0 && r.start_ms == 9.0);
  }
  // counts that are set: the launch they stand for
  for (int blocks : {1, 2, 3, 4, 9}) {
    gg::TuneSearch r;
    REQUIRE(gg::tune_search(TunePoint{blocks, 32, 77}, 640, total, [&](const TunePoint &, double t[3]) {
      t[0] = t[1] = t[2] = 1.0;
      return 0;
    }, r) == 0);
    REQUIRE(r.best.blocks == (blocks <= 2 ? 2 : 3) && r.best.chunk == 32 && r.best.batch == 77);
  }
  // a kernel with one launch shape is not timed twice
  {
    gg::TuneSearch r;
    REQUIRE(gg::tune_search(start, 288, 1, [&](const TunePoint &p, double t[3]) {
      t[0] = t[1] = t[2] = 1.0;
      return p.blocks == 2 && p.batch >= 1 ? 0 : 5;
    }, r) == 0);
    REQUIRE(r.points == 10 && r.best.blocks == 2);
  }
  // a status ends the search
  {
    gg::TuneSearch r;
    int calls = 0;
    REQUIRE(gg::tune_search(start, 640, total, [&](const TunePoint &, double t[3]) {
      t[0] = t[1] = t[2] = 1.0;
      return ++calls == 4 ? -7 : 0;
    }, r) == -7 && calls == 4);
  }
  std::puts("ok");
  return 0;
}
