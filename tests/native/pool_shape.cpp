// Launch shapes of the pooled kernels over the tables, runs and options that the entry points take.
#include <climits>
#include <cstdio>

#include "host_warp.h"

#include "../../opengate_gb300/csrc/gg_pool.cuh"

constexpr size_t kOptin = 227 * 1024;

#define REQUIRE(x)                                                                                      \
  if (!(x)) {                                                                                           \
    std::printf("line %d: %s (tables %zu, blocks %d, histories %llu, slot %zu)\n", __LINE__, #x, table, \
                blocks, (unsigned long long)n, slot);                                                   \
    return 1;                                                                                           \
  }

template <typename real>
static int check(size_t slot, int queues) {
  using Shape = gg::PoolShape<real>;
  const size_t most_table = 200 * 1024 - gg::hist_list_bytes<real>(2);  // as gg_upload_tables allows
  for (int n_sm : {1, 132, 152})
    for (size_t table : {(size_t)4096, (size_t)57344, (size_t)110000, most_table / 16 * 16})
      for (int blocks : {0, 1, 2, 3, 4, 5, INT_MAX, -1})
        for (uint64_t n : {1ull, 31ull, 33ull, 1000ull, 4864ull, 4865ull, 20000ull, 65536ull, 97280ull, 150000ull, 1ull << 26, 0xffffffffull}) {
          gg::PoolPlan p{}, q{};
          REQUIRE(gg::pool_shape<real>(n_sm, kOptin, table, blocks, n, slot, 24, queues, &p));
          REQUIRE(p.grid == n_sm && p.block >= 32 && p.block <= Shape::kBlock && p.block % 32 == 0);
          REQUIRE(p.gangs >= 1 && p.gangs <= Shape::kGangs && p.gang_threads % 32 == 0);
          REQUIRE(p.gangs * p.gang_threads >= p.block && (p.gangs - 1) * p.gang_threads < p.block);
          REQUIRE(p.slots >= 8 && p.slots <= Shape::kRing - 32);
          REQUIRE(p.smem + gg::pool_static<real>(queues) <= kOptin);
          REQUIRE(p.smem == slot * p.slots * p.gangs + table);
          REQUIRE(p.scratch == (size_t)24 * p.slots * p.gangs * n_sm);
          REQUIRE((size_t)p.slots * p.gangs * n_sm <= gg::pool_slots_most<real>(n, n_sm));
          // claims: an even share of a small run, so no gang is left out; the option's otherwise
          const uint64_t gangs = (uint64_t)p.grid * p.gangs;
          for (int chunk : {1, 64, 4096, INT_MAX}) {
            const uint64_t got = (uint64_t)gg::pool_chunk(p, chunk, n);
            const uint64_t warps = (uint64_t)std::max(p.block / 32 / p.gangs, 1);
            REQUIRE(got >= 1 && got <= (n + gangs - 1) / gangs);
            REQUIRE(got == (n + gangs - 1) / gangs || got >= std::max<uint64_t>(32, warps * std::min(chunk, 1 << 20)));
          }
          // one block of 256 threads per SM is taken as two, more than four as four
          const int same = blocks > 4 ? 4 : (blocks == 1 ? 2 : (blocks < 0 ? 0 : blocks));
          REQUIRE(gg::pool_shape<real>(n_sm, kOptin, table, same, n, slot, 24, queues, &q));
          REQUIRE(p.block == q.block && p.gangs == q.gangs && p.slots == q.slots);
          // a full run with room for its photons has its full block, or at least 512 threads
          if (table <= 57344 && n >= (uint64_t)n_sm * Shape::kBlock)
            REQUIRE(p.block >= (blocks <= 0 || blocks > 2 ? Shape::kBlock : std::min(Shape::kBlock, 512)));
        }
  return 0;
}

int main() {
  const int rc = check<float>(sizeof(gg::DoseSlot<float>), 4) || check<float>(sizeof(gg::GridSlot<float>), 4) ||
                 check<float>(sizeof(gg::TleSlot<float>), 5) || check<double>(sizeof(gg::DoseSlot<double>), 4) ||
                 check<double>(sizeof(gg::GridSlot<double>), 4) || check<double>(sizeof(gg::TleSlot<double>), 5);
  std::puts(rc ? "wrong" : "ok");
  return rc;
}
