// gg_arf.cu - ARF (angular response function) training rows on the GPU.
//
// Replaces the ARF training-dataset simulation of the reference
// (GateARFTrainingDatasetActor, core/opengate_core/opengate_lib/
// GateARFTrainingDatasetActor.cpp:76-137, with the plane source of
// contrib/spect/ge_discovery_nm670.py:994-1027): photons start on the
// collimator front face of one head, are tracked through collimator and
// crystal by the same head transport as the SPECT head stage, and each gives
// the row (E, theta, phi, w) - energy and direction at the face, and the last
// energy window containing the event's crystal energy (+1; 0 = none).  Rows
// with w = 0 are kept with probability 1 / russian_roulette.
//
// Rows come out in sample order (bit-reproducible for a seed): one kernel
// tracks one sample per thread into a staging row and counts the kept rows of
// each block of kArfBlock samples, one kernel turns the block counts into offsets, and one kernel
// compacts the kept rows.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gg_device.cuh"
#include "gg_internal.h"
#include "gg_physics.cuh"
#include "gg_spect.cuh"

namespace gg {

constexpr float kRadToDeg = 57.295779513082320876f;

// Resident blocks per SM of k_arf_sample; FP64 needs more registers.
template <typename real>
constexpr int kArfBlocks = sizeof(real) == 4 ? 6 : 3;

// Persistent: a warp takes 32 samples at a time, so none waits for the slowest
// warp of its block.  Bound by instruction issue: the photons' paths through
// the holes, septa and layers diverge (8 of 32 lanes active).  1e6 samples,
// medium-energy collimator: 306 -> 239 us with the block's barrier, the
// interactions inside the flights' loop and 4 resident blocks before; 6 / 5 /
// 4 / 3 / 2 blocks: 375 / 382 / 407 / 434 / 493 us for the whole call.
// Photons in shared-memory slots with one event kind per round (gg_pool.cuh)
// gained nothing here: 14 lanes, but twice the instructions, 301 us.
template <typename real>
__global__ void __launch_bounds__(256, kArfBlocks<real>) k_arf_sample(Scene<real> s, ArfArgs p) {
  __shared__ BlockCounters bc;
  __shared__ real sec_store[6 * 256];
  __shared__ unsigned int n_head, n_singles;
  if (threadIdx.x == 0) {
    bc = BlockCounters{0, 0, 0, 0, 0, 0, 0, 0};
    n_head = 0;
    n_singles = 0;
  }
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u;
  unsigned int steps = 0, singles = 0;
  for (;;) {
    unsigned long long i = 0;  // the warp's next 32 samples
    if (lane == 0) i = atomicAdd(p.next, 32ull);
    i = __shfl_sync(0xffffffffu, i, 0) + lane;
    if (i - lane >= p.n) break;
    bool keep = false;
    if (i < p.n) {
      Rng g;
      g.init(p.seed, p.first + i, 1u);
      Photon<real> ph;
      const real hx = (real)p.half_extent[0], hy = (real)p.half_extent[1];
      real u = R<real>(2) * u01<real>(g);
      u = u - R<real>(1);
      ph.pos[0] = u * hx;
      u = R<real>(2) * u01<real>(g);
      u = u - R<real>(1);
      ph.pos[1] = u * hy;
      ph.pos[2] = R<real>(0);
      real ct, st;
      if (p.theta_uniform) {
        const real f = u01<real>(g) * (real)p.theta_max_turn;
        gg_sincos_turn(f, st, ct);
      } else {
        real w = R<real>(1) - (real)p.cos_theta_max;
        w = u01<real>(g) * w;
        ct = R<real>(1) - w;
        real st2 = ct * ct;
        st2 = R<real>(1) - st2;
        st = gg_sqrt(st2 > R<real>(0) ? st2 : R<real>(0));
      }
      real sp, cp;
      gg_sincos_turn(u01<real>(g), sp, cp);
      ph.dir[0] = st * cp;
      ph.dir[1] = st * sp;
      ph.dir[2] = ct;
      real de = (real)p.e_max - (real)p.e_min;
      de = de * u01<real>(g);
      const real e = (real)p.e_min + de;
      float4 row;
      row.x = (float)e;
      row.y = acosf((float)ph.dir[2]) * kRadToDeg;
      row.z = atan2f((float)ph.dir[1], (float)ph.dir[0]) * kRadToDeg;
      set_energy(s, ph, e);
      ph.alive = 1;
      ph.in_head = 1;
      ph.in_image = 0;
      ph.head = 0;
      ph.hreg = 0;
      ph.left_hole = 0;
      ph.exclude = -1;
      ph.run = 0;
      ph.w = R<real>(1);
      ph.steps = 0;
      Secondary<real> sec;
      sec.base = sec_store;
      sec.stride = blockDim.x;
      sec.tid = threadIdx.x;
      sec.has = 0;
      Event<real> ev;
      ev.clear();
      for (;;) {  // flights to the next interaction, which the warp's photons then have together
        int mat;
        bool hit = false;
        while (!hit && ph.alive && ph.in_head) {
          if (++ph.steps > kStepCap) {
            atomicAdd(&bc.loop_capped, 1u);
            break;
          }
          ++steps;
          hit = head_flight(s, ph, g, mat) != 0;
        }
        if (!hit) break;
        head_interaction(s, ph, g, &bc, mat, ph.hreg == s.hreg_cr ? 2 : 3, sec, ev);
      }
      int label = 0;
      real ed = ev.esum[0];
      if (ed > R<real>(0)) {
        ++singles;
        if (s.eblur) ed = blur_energy(s, ed, g);  // the window the digitizer chain reports
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < s.n_win && ed >= s.wlo[k] && ed < s.whi[k]) label = k + 1;
      }
      row.w = (float)label;
      keep = true;
      if (label == 0) {
        const real r = u01<real>(g) * (real)p.russian_roulette;
        keep = r < R<real>(1);
      }
      if (!keep) row.w = -1.0f;
      p.stage[i] = row;
    }
    const unsigned kept = __popc(__ballot_sync(0xffffffffu, keep));
    if (lane == 0) atomicAdd(&p.block_count[i / kArfBlock], kept);
  }
  atomicAdd(&n_head, steps);
  atomicAdd(&n_singles, singles);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long *cnt = p.counters;
    if (n_head) atomicAdd(&cnt[GG_CNT_HEAD_STEPS], (unsigned long long)n_head);
    if (n_singles) atomicAdd(&cnt[GG_CNT_SINGLES], (unsigned long long)n_singles);
    if (bc.loop_capped) atomicAdd(&cnt[GG_CNT_LOOP_CAPPED], (unsigned long long)bc.loop_capped);
  }
}

// Exclusive prefix of the per-block kept counts (one block of 1024 threads; the
// counts of one launch are at most 16384).
__global__ void k_arf_offsets(const unsigned int *block_count, unsigned long long *block_off, unsigned int n_blocks,
                              unsigned long long *total) {
  __shared__ unsigned long long part[32];
  const unsigned int per = (n_blocks + blockDim.x - 1) / blockDim.x;
  const unsigned int b0 = threadIdx.x * per;
  unsigned long long sum = 0;
  for (unsigned int b = b0; b < b0 + per && b < n_blocks; ++b) sum += block_count[b];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned long long end = sum;  // inclusive prefix in the warp, then of the warps
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= (unsigned)o) end += x;
  }
  if (lane == 31u) part[warp] = end;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long own = part[lane];
    unsigned long long run = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long x = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= (unsigned)o) run += x;
    }
    const unsigned long long first = *total;
    part[lane] = first + run - own;
    __syncwarp();
    if (lane == 31u) *total = first + run;
  }
  __syncthreads();
  unsigned long long off = part[warp] + end - sum;
  for (unsigned int b = b0; b < b0 + per && b < n_blocks; ++b) {
    block_off[b] = off;
    off += block_count[b];
  }
}

// Kept rows to their place: block offset + rank of the row inside its block.
__global__ void __launch_bounds__(kArfBlock) k_arf_compact(const float4 *stage, const unsigned long long *block_off,
                                                     uint64_t n, float4 *rows, uint64_t capacity) {
  __shared__ unsigned int warp_base[kArfBlock / 32];
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float4 r = make_float4(0.f, 0.f, 0.f, -1.f);
  if (i < n) r = stage[i];
  const bool keep = i < n && r.w >= 0.0f;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) warp_base[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int run = 0;
    for (int k = 0; k < kArfBlock / 32; ++k) {
      const unsigned int v = warp_base[k];
      warp_base[k] = run;
      run += v;
    }
  }
  __syncthreads();
  if (keep) {
    const uint64_t dst = block_off[blockIdx.x] + warp_base[warp] + __popc(m & ((1u << lane) - 1u));
    if (dst < capacity) rows[dst] = r;
  }
}

template <typename real>
cudaError_t launch_arf_dataset(const Scene<real> &s, const ArfArgs &p, int n_sm, float4 *rows, uint64_t capacity,
                               unsigned long long *total, cudaStream_t st) {
  const unsigned int blocks = (unsigned int)((p.n + kArfBlock - 1) / kArfBlock);
  if (blocks == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(p.next, 0, sizeof(unsigned long long), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(p.block_count, 0, blocks * sizeof(unsigned int), st);
  if (e != cudaSuccess) return e;
  k_arf_sample<real><<<std::min(blocks, (unsigned)(n_sm * kArfBlocks<real>)), 256, 0, st>>>(s, p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_arf_offsets<<<1, 1024, 0, st>>>(p.block_count, p.block_off, blocks, total);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_arf_compact<<<blocks, kArfBlock, 0, st>>>(p.stage, p.block_off, p.n, rows, capacity);
  return cudaGetLastError();
}

template cudaError_t launch_arf_dataset<float>(const Scene<float> &, const ArfArgs &, int, float4 *, uint64_t,
                                               unsigned long long *, cudaStream_t);
template cudaError_t launch_arf_dataset<double>(const Scene<double> &, const ArfArgs &, int, float4 *, uint64_t,
                                                unsigned long long *, cudaStream_t);

}  // namespace gg
