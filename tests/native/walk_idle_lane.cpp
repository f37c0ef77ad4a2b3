// A walk round of the track-length estimator in which the lane has no slot and slot 0 has never held
// a photon: its shared memory is whatever was there.  The tables end at a page that may not be read.
#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "host_warp.h"

#include "../../opengate_gb300/csrc/gg_pool.cuh"

// n elements that end where unreadable pages begin (more of them than a 16-bit index can skip)
template <typename T>
static T *guarded(size_t n) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), guard = ((size_t)1 << 17) * sizeof(double);
  const size_t room = (n * sizeof(T) + page - 1) / page * page;
  char *p = (char *)mmap(nullptr, room + guard, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == (char *)MAP_FAILED || mprotect(p + room, guard, PROT_NONE) != 0) std::exit(2);
  return (T *)(p + room) - n;
}

template <typename real>
static int check() {
  constexpr int kE = 16, kMat = 2;
  gg::Scene<real> s{};
  s.n_e = kE;
  s.n_comp = kMat;
  s.n_mat = kMat;
  s.nx = 4;
  s.ny = s.nz = 1;
  for (int a = 0; a < 3; ++a) {
    s.bmin[a] = 0;
    s.sp[a] = s.inv_sp[a] = 1;
  }
  real *muen = guarded<real>(kMat * kE), *rho = guarded<real>(kMat);
  int *comp = guarded<int>(kMat);
  uint16_t *labels = guarded<uint16_t>(4);
  for (int i = 0; i < kMat * kE; ++i) muen[i] = real(1);
  for (int m = 0; m < kMat; ++m) {
    comp[m] = m;
    rho[m] = real(1);
  }
  for (int v = 0; v < 4; ++v) labels[v] = (uint16_t)(v & 1);
  s.muen = muen;
  s.mat_rho = rho;
  s.mat_comp = comp;
  s.labels = labels;
  std::vector<unsigned long long> acc(4), acc2(8);
  const gg::Tally<real> t{acc.data(), acc2.data()};
  static gg::TleSlot<real> slots[2];
  unsigned n_dep = 0, n_ent = 0, n_over = 0;
  for (int fill = 0; fill < 256; fill += 15) {  // what the shared memory held
    std::memset(slots, fill, sizeof(slots));
    for (auto &S : slots) S.e = make_uint4(0u, 0u, 0u, 0u);  // all that a kernel clears
    if (gg::tle_walk<real>(s, slots, -1, 0u, t, n_dep, n_ent, n_over) != gg::kQNone) return 1;
  }
  if (n_dep || n_ent || n_over) return 1;
  // a photon in slot 1 walks from the first voxel through the third: 1.5 voxels' path scored
  gg::TleSlot<real> &S = slots[1];
  S.a = {real(0.5), real(0.5), real(0.5), real(10)};
  S.b = {real(1), real(0), real(0), real(2)};
  S.c = {real(1), real(1), real(0), gg::bits_real(real(0), (uint32_t)(kE - 2))};
  gg::VoxelWalk<real> w;
  const real p[3] = {S.a.x, S.a.y, S.a.z}, d[3] = {S.b.x, S.b.y, S.b.z};
  w.start(s, p, d);
  gg::tle_store(S.x, w, real(1.75));
  if (gg::tle_walk<real>(s, slots, 1, 0u, t, n_dep, n_ent, n_over) != gg::kQFly) return 1;
  const int n = (int)((S.e.z >> gg::kSlList) & 15u);
  if (n != 3 || n_dep != 3u) return 1;
  const real want[3] = {real(1), real(2), real(0.5)};  // energy 2, coefficient 1
  for (int k = 0; k < 3; ++k)
    if (S.x.vox[k] != (uint32_t)k || S.x.acc[k] != want[k]) return 1;
  return 0;
}

int main() {
  const int rc = check<float>() || check<double>();
  std::puts(rc ? "wrong" : "ok");
  return rc;
}
