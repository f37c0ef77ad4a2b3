// gg_spect.cu - SPECT acquisition as a two-stage wavefront.
//
// A SPECT history crosses three very different kinds of geometry: the
// voxelised phantom (Woodcock steps and label gathers), the air of the world,
// and the heads (collimator hole lattice, crystal and the digitizer event).
// One kernel that carries all three keeps every warp's lanes spread over the
// three code paths.  Here the work is split by where the photon is:
//
//   * phantom stage: source records (or photons handed back by the head
//     stage) are tracked in the image and the world; a photon that reaches a
//     head box is written, with its RNG position and event, to the head queue
//     and its lane takes the next history;
//   * head stage: queued photons are tracked through collimator, gap and
//     crystal (and the world between the heads); the event is scored into the
//     projection when the photon dies; a photon that flies back into the
//     image is written to the return queue for another phantom pass.
//
// The host alternates the stages until the return queue stays empty.  Every
// photon executes the same operations in the same order as in a single
// kernel (the queues only change which lane runs them), so projections and
// counters equal those of the CPU oracle bit for bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_device.cuh"
#include "gg_internal.h"
#include "gg_physics.cuh"
#include "gg_pool.cuh"
#include "gg_queue.cuh"
#include "gg_spect.cuh"
#include "gg_split.h"

namespace gg {

// Free-flight modes of the stages (Scene::ff).
constexpr int kFfPrimary = 1, kFfScatter = 2;

// Head-stage flight: one step in a head, or one world step; a photon whose
// world step ends at the image-box entry leaves the stage (kPush).
template <typename real, bool FF>
__device__ __forceinline__ int head_stage_flight(const Scene<real> &s, Photon<real> &ph, Rng &g, BlockCounters *bc,
                                                 int &pmat, int &pscored, unsigned int &n_world,
                                                 unsigned int &n_head) {
  if (++ph.steps > kStepCap) {
    atomicAdd(&bc->loop_capped, 1u);
    ph.alive = 0;
    return kRefill;
  }
  if (ph.in_head) {
    ++n_head;
    int mat;
    if (head_flight(s, ph, g, mat)) {
      pmat = mat;
      pscored = ph.hreg == s.hreg_cr ? 2 : 3;
      return kInteract;
    }
    return ph.alive ? kFly : kRefill;  // (stopped by a shielded side)
  }
  ++n_world;
  if constexpr (FF) {  // free flight to another head (the image crossed on the way)
    if (ff_flight(s, ph, R<real>(-2))) return kFly;
    atomicAdd(&bc->escaped, 1u);
    return kRefill;
  }
  if (spect_world_flight(s, ph, g)) {
    pmat = s.world_mat;
    pscored = 0;
    return kInteract;
  }
  if (!ph.alive) {
    atomicAdd(&bc->escaped, 1u);
    return kRefill;
  }
  return ph.in_image ? kPush : kFly;
}

// Block counters and per-lane step counts into the global counters.
__device__ __forceinline__ void stage_counters(unsigned long long *cnt, const BlockCounters &bc, unsigned lane,
                                               unsigned int n_wood, unsigned int n_real, unsigned int n_world,
                                               unsigned int n_head, unsigned int n_singles) {
  auto warp_add = [&](unsigned int v, int slot) {
    unsigned long long x = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0 && x) atomicAdd(&cnt[slot], x);
  };
  warp_add(n_wood, GG_CNT_WOODCOCK_STEPS);
  warp_add(n_real, GG_CNT_REAL_INTERACTIONS);
  warp_add(n_world, GG_CNT_WORLD_STEPS);
  warp_add(n_head, GG_CNT_HEAD_STEPS);
  warp_add(n_singles, GG_CNT_SINGLES);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bc.escaped) atomicAdd(&cnt[GG_CNT_ESCAPED], (unsigned long long)bc.escaped);
    if (bc.loop_capped) atomicAdd(&cnt[GG_CNT_LOOP_CAPPED], (unsigned long long)bc.loop_capped);
    if (bc.stack_overflow) atomicAdd(&cnt[GG_CNT_STACK_OVERFLOW], (unsigned long long)bc.stack_overflow);
    if (bc.secondaries) atomicAdd(&cnt[GG_CNT_SECONDARIES], (unsigned long long)bc.secondaries);
    if (bc.list_overflows) atomicAdd(&cnt[GG_CNT_LIST_OVERFLOWS], (unsigned long long)bc.list_overflows);
  }
}

// Largest cosine that a photon scattered by theta (cos, sin) can make with a
// head axis u over the azimuth: cos(theta - theta_u) = cos(theta) c0 + sin(theta)
// s0, c0 = d.u, s0 = sqrt(1 - c0^2).  A copy whose cosine stays below the angle
// check of every head (ff_target) is dropped before its azimuth is drawn; a
// margin of 1e-4 keeps every direction the full check would accept (rounding is
// far below it), so that changes no result.
template <typename real>
__device__ __forceinline__ real axis_sine(real c0) {
  const real s0 = R<real>(1) - c0 * c0;
  return gg_sqrt(s0 > R<real>(0) ? s0 : R<real>(0));
}

template <typename real>
__device__ __forceinline__ bool cone_reachable(const Scene<real> &s, int run, const real d[3], real cost, real sint2,
                                               real cos_min) {
  const real sint = gg_sqrt(sint2 > R<real>(0) ? sint2 : R<real>(0));
  const real lim = cos_min - R<real>(1e-4);
  for (int h = 0; h < s.n_heads; ++h) {
    const HeadFrame<real> f = head_frame(s, run, h);
    const real c0 = dot3(d, f.u);
    real m = cost * c0;
    m = m + sint * axis_sine(c0);
    if (!(m < lim)) return true;
  }
  return false;
}

// Words p .. p + 3 of a stream, p = 3 t: a trial's three draws, and the azimuth
// drawn after it when it is accepted.  w3: word 3, when t = 1 (kept from the
// first trial, so that the second makes one block too).
struct TrialWords {
  uint32_t w[4];

  __device__ __forceinline__ void draw(uint32_t t, uint32_t w3, uint32_t stream, uint32_t h0, uint32_t h1, uint32_t k0,
                                       uint32_t k1) {
    const uint32_t p = 3u * t, at = p & 3u;
    // (in line: the round keys of the launch's seed stay in uniform registers)
    uint32_t ctr[4] = {(p >> 2) + (t == 1u ? 1u : 0u), stream, h0, h1}, o[4];
    philox4x32_10(ctr, k0, k1, o);
    uint4 a = make_uint4(o[0], o[1], o[2], o[3]), b = a;
    if (t == 1u) a.w = w3;
    else if (at != 0u) b = philox_block((p >> 2) + 1u, stream, h0, h1, k0, k1);
    w[0] = at == 0u ? a.x : (at == 1u ? a.y : (at == 2u ? a.z : a.w));
    w[1] = at == 0u ? a.y : (at == 1u ? a.z : (at == 2u ? a.w : b.x));
    w[2] = at == 0u ? a.z : (at == 1u ? a.w : (at == 2u ? b.x : b.y));
    w[3] = at == 0u ? a.w : (at == 1u ? b.x : (at == 2u ? b.y : b.z));
  }
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// What is certain about a Klein-Nishina trial and the direction it leads to from
// approximate arithmetic (hardware exp2, reciprocal, square root: relative
// errors at most 2^-22, 2^-23, 2^-23; sine, cosine: absolute 2^-20.5):
//   kTrialRejected  KleinNishina::trial() rejects it;
//   kTrialDropped   it is accepted, and the copy dies below the energy cut;
//   kTrialMissed    it is accepted above the cut, and the new direction fails the
//                   angle check against every head axis (ff_target());
//   kTrialUnsure    anything else: the exact trial decides.
// eps carries a relative error below 1.5e-6 (the exponent is at most ln(1 + 2k) <
// 2 below 1.022 MeV: its rounding adds 7e-7), so 1 - cos = (1 - eps) / (eps k)
// one below 1.5e-6 / (eps k) + 1e-6, 1 / (eps k) <= 2 + 1 / k; sin^2 twice and the
// acceptance function once that.  tol = 4e-6 (2 + 1 / k) covers each with a factor
// of two; the sine lies between those of sin^2 - 2 tol and sin^2 + 2 tol, and 2e-5
// covers the azimuth's sine and cosine and the exact check's own rounding.
enum : int { kTrialRejected = 0, kTrialDropped = 1, kTrialMissed = 2, kTrialUnsure = 3 };

struct TrialFilter {
  float k, eps0sq, alpha1, alpha2, e, tol;
  // the head axes in the scattering frame of rotate_dir(): along the direction,
  // and along its two transverse axes (azimuth 0 and a quarter turn)
  float c0[2], a1[2], a2[2];

  __device__ __forceinline__ int operator()(const uint32_t w[4], float e_min, float cos_min, bool check) const {
    constexpr float kU = 5.9604644775390625e-08f;
    const float r0 = (float)(w[0] >> 8) * kU, r1 = (float)(w[1] >> 8) * kU, r2 = (float)(w[2] >> 8) * kU;
    const float d = alpha1 - alpha2 * r0;
    const float sq = fmaf(1.0f - eps0sq, r1, eps0sq);
    const bool log_part = d > 0.0f;
    const float eps = log_part ? fast_exp2(alpha1 * r1 * -1.44269504f) : fast_sqrt(sq);
    const float epssq = log_part ? eps * eps : sq;
    const float onecost = (1.0f - eps) * fast_rcp(eps * k);
    const float sint2 = onecost * (2.0f - onecost);
    const float gr = 1.0f - eps * sint2 * fast_rcp(1.0f + epssq);
    const float ed = eps * e;
    if (fabsf(d) < 1e-5f * alpha1 || !(fabsf(gr - r2) > tol) || fabsf(ed - e_min) < 1e-5f * e_min) return kTrialUnsure;
    if (gr < r2) return kTrialRejected;
    if (ed < e_min) return kTrialDropped;
    if (!check) return kTrialUnsure;
    const float phi = (float)(w[3] >> 8) * (kU * 6.28318531f) - 3.14159265f;  // (half a turn off: the signs below)
    const float cp = __cosf(phi), sp = __sinf(phi);
    const float cost = 1.0f - onecost, hi = fast_sqrt(fmaxf(sint2 + 2.0f * tol, 0.0f)),
                lo = fast_sqrt(fmaxf(sint2 - 2.0f * tol, 0.0f));
    bool miss = true;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float t = -(cp * a1[h] + sp * a2[h]);
      miss = miss && fmaf(cost, c0[h], (t > 0.0f ? hi : lo) * t) + tol + 2e-5f < cos_min;
    }
    return miss ? kTrialMissed : kTrialUnsure;
  }
};

// What a warp of the split kernel keeps in shared memory.
constexpr int kSplitBatch = 32;  // requests at a time
struct SplitWarp {
  TrialFilter f[kSplitBatch];  // the requests' constants, and their streams
  uint32_t h0[kSplitBatch], h1[kSplitBatch], stream[kSplitBatch];
  // copies rejected so far, waiting for their next trial: copy of the batch | trial << 20
  uint32_t retry[kSplitRetry], word3[kSplitRetry];  // (word 3 of its stream)
  // copies of the batch whose trial the filter leaves open: copy | trial << 20
  uint32_t open[kSplitOpen];
};
static_assert(GG_MAX_SPLITTING * kSplitBatch < (1 << 20) && kLoopCap < (1 << 12), "a retry packs copy and trial");

// Scatter splitting, the copies (GateScatterSplittingFreeFlightOptn.cpp:69-149).
// Request r of the phantom stage holds the photon before a Compton (or
// Rayleigh) interaction; its copy c re-samples that interaction from there on
// Philox stream 2 + base + c of the history, with 1 / n of the weight, and flies
// freely to a head: the intersection check of the angular acceptance is the
// flight itself (a copy that misses every head cannot be detected), the angle
// check comes before the optical depth.  A copy whose line enters a head (past
// the checks) goes to the walk queue (q.out_q), where k_spect_walk computes its
// optical depth.  Compton requests fill the buffer from the front and Rayleigh
// requests from the back; when together they overflowed it, nothing is done
// (the host repeats the pass on fewer histories).
//
// A warp takes 32 Compton requests: each lane computes one request's constants
// for all its copies, then the lanes run the copies one trial at a time.  Trial
// t of a copy draws words 3t .. 3t + 2 of its stream, so a copy needs no state
// but t between trials: rejected ones wait until 32 such fill a round.  Nearly
// every trial is settled by approximate arithmetic (TrialFilter); the others
// wait for a round of the exact trial, the rest of the scattering and the head
// checks, whose arithmetic and draws are those of the plain sequence.
// Bound by instruction issue (70 % active, 25.6 lanes): 2.2e8 copies at 140 keV 9 ->
// 4.1 ms against one thread per copy from request to end; of that, constants per
// request and full rounds 6.6, the approximate trial with the azimuth 4.3, the
// generator in line 4.1.
// Three resident blocks (80 registers) in FP32: with 84 registers only two fit, 6.17
// -> 6.50 ms for the copies and walks of 1e7 decays' scatter pass at 140 keV.
template <typename real>
__global__ void __launch_bounds__(256, sizeof(real) == 4 ? 3 : 2) k_spect_split(Scene<real> s, KernelArgs args, StageArgs q) {
  __shared__ BlockCounters bc;
  __shared__ SplitWarp warps[kBlock / 32];
  if (threadIdx.x == 0) bc = BlockCounters{0, 0, 0, 0, 0, 0, 0, 0};
  __syncthreads();
  const uint64_t n_c = *q.split_n, n_r = q.split_n[1];
  if (n_c + n_r > (uint64_t)q.split_cap) return;
  const SplitQueue<real> sq = SplitQueue<real>::carve(q.split_q, q.split_cap);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  SplitWarp &P = warps[threadIdx.x >> 5];
  const uint32_t k0 = (uint32_t)args.seed, k1 = (uint32_t)(args.seed >> 32);
  const bool check = s.ss_cos > R<real>(-1);
  const float cos_min = (float)s.ss_cos, e_min = (float)s.e_min;
  unsigned int n_world = 0, n_esc = 0;

  // Request r's photon before the interaction, its copy c's stream.
  auto load_copy = [&](size_t r, uint32_t c, int n, Photon<real> &cp, Rng &g) {
    cp.pos[0] = sq.px[r];
    cp.pos[1] = sq.py[r];
    cp.pos[2] = sq.pz[r];
    cp.dir[0] = sq.dx[r];
    cp.dir[1] = sq.dy[r];
    cp.dir[2] = sq.dz[r];
    cp.e = sq.e[r];
    cp.w = sq.w[r] / (real)n;
    cp.alive = 1;
    cp.run = sq.run[r];
    const uint64_t hid = sq.hid[r];
    g.init(args.seed, hid, 2u + sq.base[r] + c);
    return hid;
  };
  // A scattered copy's head checks and its place in the walk queue (every lane of the warp calls it).
  auto to_walk = [&](bool live, Photon<real> &cp, const Rng &g, uint64_t hid) {
    bool push = false;
    if (live) {
      cp.exclude = -1;
      cp.steps = 0;
      cp.head = 0;
      cp.hreg = 0;
      ++n_world;
      real tb;
      push = ff_target(s, cp, s.ss_cos, tb) != 0;  // with the angle check of the angular acceptance
      if (!push) ++n_esc;
    }
    const size_t kq = queue_claim(q.out_n, push, lane, lt_mask);
    if (push && kq < q.q_cap) {
      real v[kEvSlots];
      queue_put<real, true>(out, kq, cp, g, hid, v, false);
    }
  };

  const uint64_t n_warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  // ---- Compton requests, `batch` at a time (fewer when there are not enough for all warps)
  const uint32_t per = (uint32_t)s.ss_nc;
  const uint32_t batch = (uint32_t)min((uint64_t)kSplitBatch, max(n_c / n_warps, (uint64_t)1));
  const uint32_t step_r = per ? 32u / per : 0u, step_c = per ? 32u % per : 0u;  // 32 copies on
  for (uint64_t r0 = warp * batch; per && r0 < n_c; r0 += n_warps * batch) {
    const uint32_t nb = (uint32_t)min((uint64_t)batch, n_c - r0);
    if (lane < nb) {
      const uint64_t r = r0 + lane;
      const uint64_t hid = sq.hid[r];
      const real d[3] = {sq.dx[r], sq.dy[r], sq.dz[r]};
      const KleinNishina<real> kn(sq.e[r]);
      TrialFilter f;
      f.k = (float)kn.k;
      f.eps0sq = (float)kn.eps0sq;
      f.alpha1 = (float)kn.alpha1;
      f.alpha2 = (float)kn.alpha2;
      f.e = (float)sq.e[r];
      f.tol = 4e-6f * (2.0f + 1.0f / f.k);
      const int run = sq.run[r];
      real t1[3] = {R<real>(1), R<real>(0), R<real>(0)}, t2[3] = {R<real>(0), R<real>(1), R<real>(0)};
      const real pp = gg_sqrt(d[0] * d[0] + d[1] * d[1]);
      if (pp > R<real>(1e-4)) {
        t1[0] = d[0] * d[2] / pp;
        t1[1] = d[1] * d[2] / pp;
        t1[2] = -pp;
        t2[0] = -d[1] / pp;
        t2[1] = d[0] / pp;
      } else {
        f.tol = 4.0f;  // (along z: rounding of the frame counts; the exact trial decides)
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // (one head: twice the same)
        const HeadFrame<real> fr = head_frame(s, run, h < s.n_heads ? h : 0);
        f.c0[h] = (float)dot3(d, fr.u);
        f.a1[h] = (float)dot3(t1, fr.u);
        f.a2[h] = (float)dot3(t2, fr.u);
      }
      P.f[lane] = f;
      P.h0[lane] = (uint32_t)hid;
      P.h1[lane] = (uint32_t)(hid >> 32);
      P.stream[lane] = 2u + sq.base[r];
    }
    __syncwarp();
    const uint32_t total = nb * per;
    uint32_t next = 0;                               // copies not begun
    uint32_t fr = lane / per, fc = lane - fr * per;  // request and copy of copy next + lane
    int nr = 0, no = 0;                              // copies waiting in P.retry, P.open (the same in every lane)
    for (;;) {
      const SplitRound round = split_round(nr, no, next >= total);
      if (round == kSplitDone) break;
      if (round == kSplitExactTrials) {
        const int n = min(no, 32);
        no -= n;
        bool live = false, again = false;
        uint32_t id = 0, w3 = 0;
        Photon<real> cp;
        Rng g;
        uint64_t hid = 0;
        if ((int)lane < n) {
          id = P.open[no + (int)lane];
          const uint32_t t = id >> 20, r = (id & 0xfffffu) / per;
          hid = load_copy((size_t)(r0 + r), (id & 0xfffffu) - r * per, s.ss_nc, cp, g);
          // the stream after 3t words: the state an Rng reaches by drawing them
          const uint32_t p = 3u * t;
          if ((p & 3u) == 0u) {
            g.blk = p >> 2;
          } else {
            const uint4 b = philox_block(p >> 2, g.stream, g.h0, g.h1, g.k0, g.k1);
            g.buf[0] = b.x;
            g.buf[1] = b.y;
            g.buf[2] = b.z;
            g.buf[3] = b.w;
            g.blk = (p >> 2) + 1u;
            g.idx = (int)(p & 3u);
          }
          const KleinNishina<real> kn(cp.e);
          real eps, onecost, sint2;
          bool done = kn.trial(g, eps, onecost, sint2);
          w3 = g.buf[3];  // (after a first trial: word 3)
          if (!done && t + 1u >= (uint32_t)kLoopCap) {
            atomicAdd(&bc.loop_capped, 1u);
            done = true;
          }
          again = !done;
          id += 1u << 20;
          if (done && !(eps * cp.e < s.e_min)) {  // (below the energy cut the copy dies)
            live = !check || cone_reachable(s, cp.run, cp.dir, R<real>(1) - onecost, sint2, s.ss_cos);
            if (live) {
              scatter_dir(cp, g, R<real>(1) - onecost, sint2);
              cp.e = eps * cp.e;  // (the walk kernel sets its energy-grid state)
            } else {              // a live copy that fails the head checks, as counted there
              ++n_world;
              ++n_esc;
            }
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, again);
        if (again) {
          P.retry[nr + __popc(m & lt_mask)] = id;
          P.word3[nr + __popc(m & lt_mask)] = w3;
        }
        nr += __popc(m);
        to_walk(live, cp, g, hid);
        __syncwarp();
        continue;
      }
      // ---- a round of filtered trials: of rejected copies, or first ones
      bool on;
      uint32_t r = 0, c = 0, t = 0, w3 = 0;
      if (round == kSplitRetries) {
        const int n = min(nr, 32);
        nr -= n;
        on = (int)lane < n;
        if (on) {
          const uint32_t id = P.retry[nr + (int)lane];
          w3 = P.word3[nr + (int)lane];
          t = id >> 20;
          r = (id & 0xfffffu) / per;
          c = (id & 0xfffffu) - r * per;
        }
      } else {
        on = next + lane < total;
        r = on ? fr : 0u;
        c = fc;
        next += 32u;
        fr += step_r;
        fc += step_c;
        if (fc >= per) fc -= per, ++fr;
      }
      __syncwarp();
      int res = kTrialDropped;
      if (on) {
        TrialWords g;
        g.draw(t, w3, P.stream[r] + c, P.h0[r], P.h1[r], k0, k1);
        w3 = g.w[3];
        res = P.f[r](g.w, e_min, cos_min, check);
        if (res == kTrialRejected && t + 1u >= (uint32_t)kLoopCap) res = kTrialUnsure;
        if (res == kTrialMissed) {  // a live copy that fails the head checks, as counted there
          ++n_world;
          ++n_esc;
        }
      }
      const unsigned mr = __ballot_sync(0xffffffffu, res == kTrialRejected);
      const unsigned mo = __ballot_sync(0xffffffffu, res == kTrialUnsure);
      const uint32_t id = (r * per + c) | (t << 20);
      if (res == kTrialRejected) {
        P.retry[nr + __popc(mr & lt_mask)] = id + (1u << 20);
        P.word3[nr + __popc(mr & lt_mask)] = w3;
      }
      if (res == kTrialUnsure) P.open[no + __popc(mo & lt_mask)] = id;
      nr += __popc(mr);
      no += __popc(mo);
      __syncwarp();
    }
  }
  // ---- Rayleigh requests: one thread per copy (their copies are few)
  const uint64_t per_r = (uint64_t)s.ss_nr, all_r = n_r * per_r;
  for (uint64_t i0 = warp * 32u; i0 < all_r; i0 += n_warps * 32u) {
    const uint64_t i = i0 + lane;
    bool live = false;
    Photon<real> cp;
    Rng g;
    uint64_t hid = 0;
    if (i < all_r) {
      const uint64_t req = i / per_r;
      const size_t r = q.split_cap - 1 - (size_t)req;
      hid = load_copy(r, (uint32_t)(i - req * per_r), s.ss_nr, cp, g);
      cp.ei = energy_index(s, cp.e);
      const real cost = rayleigh_cost(s, sq.comp[r], cp, g, &bc);
      live = !check || cone_reachable(s, cp.run, cp.dir, cost, rayleigh_sint2(cost), s.ss_cos);
      if (live) {
        rayleigh_finish(cp, g, cost);
      } else {
        ++n_world;
        ++n_esc;
      }
    }
    to_walk(live, cp, g, hid);
  }
  if (n_esc) atomicAdd(&bc.escaped, n_esc);
  stage_counters(args.counters, bc, lane, 0u, 0u, n_world, 0u, 0u);
}

// Label gathers in flight per lane in the walk kernel's optical depths.
constexpr int kWalkGroup = 8;

// Free flights that passed their checks (the copies of scatter splitting
// after the split kernel, the photons of primary free flight after the
// phantom stage): the whole ff_flight (its first part again, bit for bit the
// same, then the optical depth along the line), one photon per thread, so a
// warp walks 32 lines at once instead of one line among lanes that have
// finished; photons that reach their head go to the head queue.
template <typename real>
__global__ void __launch_bounds__(256) k_spect_walk(Scene<real> sg, KernelArgs args, StageArgs q) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  Scene<real> s = sg;
  stage_tables(sg, s, smem_raw, bc);
  const uint64_t n = min((uint64_t)*q.in_n, (uint64_t)q.q_cap);
  const PQueue<real> in = PQueue<real>::carve(q.in_q, q.q_cap);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = i0 + threadIdx.x;
    Photon<real> cp;
    Rng g;
    uint64_t hid = 0;
    bool push = false, has_ev = false;
    if (i < n) {
      hid = queue_get<real, true>(s, in, i, cp, g, args.seed, has_ev);
      push = ff_flight<real, kWalkGroup>(s, cp, s.ss_cos) != 0;
      if (!push) atomicAdd(&bc.escaped, 1u);
    }
    const size_t k = queue_claim(q.out_n, push, lane, lt_mask);
    if (push) {
      if (k < q.q_cap) {
        real v[kEvSlots];
        if (has_ev) load_event(in, i, v);
        queue_put<real, true>(out, k, cp, g, hid, v, has_ev);
      } else {
        atomicOr(args.status, kStatusQueueOverflow);
      }
    }
  }
  stage_counters(args.counters, bc, lane, 0u, 0u, 0u, 0u, 0u);
}

// The phantom stage's part of a slot: x the input-queue flag (1: the photon
// came back from a head and carries an event), y its queue entry, z split
// copies of the history so far, w Compton interactions of the analog track.
template <typename real>
struct PhantomPart {
  uint4 v;
};
template <>
struct PhantomPart<float> {
  uint4 v, pad;
};
template <typename real>
using PhantomSlot = PhotonSlot<real, PhantomPart<real>>;
static_assert(sizeof(PhantomSlot<float>) % 32 == 16 && sizeof(PhantomSlot<double>) % 32 == 16, "odd 16-byte stride");

// The event of a photon that came back from a head and died in the phantom
// (out of line: less than 1 % of the photons).
template <typename real>
static __device__ __noinline__ unsigned score_returned(const Scene<real> &s, void *in_q, size_t q_cap, uint32_t entry,
                                                       int run, Rng g) {
  const PQueue<real> in = PQueue<real>::carve(in_q, q_cap);
  Event<real> ev;
  real v[kEvSlots];
  load_event(in, entry, v);
  event_from(v, ev);
  return score_singles(s, ev, run, g);
}

// Phantom stage: the pooled event loop of gg_pool.cuh (as the dose transport).
// Input: the batch's primary records (q.in_q == null) or the return queue;
// output: the head queue.  Events: a new photon, a Woodcock step in the image,
// a flight in the world (to a head box: the photon leaves the stage), an
// interaction.  SPLIT (scatter splitting): photons that reach a head die
// there, and every Compton up to the maximum level and every Rayleigh
// scattering asks for split copies (GateScatterSplittingFreeFlightOptrActor.cpp:
// 291-360), made by the split kernel.
// Bound by instruction issue and latency (46 % of issue slots, 21 active lanes):
// Tc-99m in the CT phantom, 3e7 decays, 25.0 -> 12.5 ms against one photon per thread with
// block-wide phases.
template <typename real, bool SPLIT>
__global__ void __launch_bounds__(PoolShape<real>::kBlock, 1)
    k_spect_phantom(const __grid_constant__ Scene<real> sg, KernelArgs args, StageArgs q, int n_slots,
                    int gang_threads) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  using Shape = PoolShape<real>;
  constexpr int kGangs = Shape::kGangs;
  __shared__ __align__(16) unsigned push[kGangs][3 * kQueues];
  __shared__ __align__(16) uint32_t ahead[Shape::kBlock][4];  // EventRng's second block of each thread
  __shared__ uint16_t ring[kGangs][kQueues * Shape::kRing];
  __shared__ unsigned long long s_claim[kGangs];
  Scene<real> s = sg;
  const unsigned lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  const int gang = (int)threadIdx.x / gang_threads, gang0 = gang * gang_threads;
  const int gangs = ((int)blockDim.x + gang_threads - 1) / gang_threads;
  // dynamic shared memory: slots of the gangs, tables
  PhantomSlot<real> *const slots = reinterpret_cast<PhantomSlot<real> *>(smem_raw) + gang * n_slots;
  EventQueues<Shape::kRing> Q;
  Q.init(gang, threadIdx.x - (unsigned)gang0, min((unsigned)gang_threads, blockDim.x - (unsigned)gang0), ring[gang], push[gang],
         (unsigned)n_slots);
  for (int i = (int)Q.tid; i < n_slots; i += (int)Q.size) {
    slots[i].e = make_uint4(0u, 0u, 0u, 0u);
    slots[i].x.v = make_uint4(0u, 0u, 0u, 0u);
  }
  stage_tables(sg, s, smem_raw + sizeof(PhantomSlot<real>) * (size_t)(gangs * n_slots), bc);

  const bool from_queue = !SPLIT && q.in_q != nullptr;
  const Records<real> rec = Records<real>::carve(args.records, args.rec_cap);
  PQueue<real> in{};
  if (from_queue) in = PQueue<real>::carve(q.in_q, q.q_cap);
  // a queue length above the capacity means entries were dropped (status
  // GG_ERR_QUEUE_OVERFLOW): never read past the capacity
  const uint32_t n_items =
      (uint32_t)(from_queue ? min((uint64_t)*q.in_n, (uint64_t)q.q_cap) : args.h_end - args.h_begin);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const uint32_t slot0 = (blockIdx.x * (uint32_t)gangs + (uint32_t)gang) * (uint32_t)n_slots;
  Secondary<real> sec;
  sec.base = reinterpret_cast<real *>(args.slot_scratch);
  sec.stride = (int)(gridDim.x * (uint32_t)(gangs * n_slots));
  const uint32_t k0 = (uint32_t)args.seed, k1 = (uint32_t)(args.seed >> 32);
  unsigned int n_wood = 0, n_real = 0, n_world = 0, n_singles = 0, n_esc = 0;
  ItemClaims claims;
  claims.init();

  for (;;) {
    int k;
    unsigned n;
    const int event = Q.round(k, n);
    if (event == kQNone) break;
    if (event == kQRefill) claims.take(Q, n, args.next, args.chunk, n_items, &s_claim[gang]);
    int dest = kQNone, idx = 0, kind = 0, copies = 0, pmat = 0;
    int smat = 0, pscored = 0;
    uint32_t pv = 0, trials = 0;
    bool leave = false;                               // to the head queue
    bool fresh = event != kQFly && event != kQWorld;  // direction and energy change
    bool live = k >= 0;                               // the slot holds a photon
    Photon<real> ph;
    sec.has = 0;
    uint4 e = make_uint4(0u, 0u, 0u, 0u), x = make_uint4(0u, 0u, 0u, 0u);
    uint64_t hid = 0;
    if (k >= 0) {
      PhantomSlot<real> &S = slots[k];
      e = S.e;
      x = S.x.v;
      ph.alive = 1;
      uint32_t cw = 0;
      bool aim = false;  // its path to the image boundary is not known (in a slot: negative)
      uint32_t *const buf = &S.rng.x;
      if (event == kQRefill) {
        if (!SPLIT && x.x) {
          hid = args.h_begin + e.y;
          Rng g;
          rng_resume(g, args.seed, hid, (e.x << 3) | ((e.z >> kSlIdx) & 7u), S.rng);
          n_singles += score_returned(sg, q.in_q, q.q_cap, x.y, (int)e.w, g);
        }
        uint32_t h;
        const bool have = claims.item(Q.tid, h);
        uint32_t f = kRecDead;
        size_t r = h;
        if (!from_queue) r += args.h_begin - args.rec_first;  // record of the history
        if (have) f = from_queue ? kRecInImage : rec.flags[r];
        dest = have || !claims.exhausted ? kQRefill : kQNone;
        live = (f & 3u) != kRecDead;
        e = x = make_uint4(0u, 0u, 0u, 0u);
        if (live) {
          const real *const src[7] = {from_queue ? in.px : rec.px, from_queue ? in.py : rec.py,
                                      from_queue ? in.pz : rec.pz, from_queue ? in.dx : rec.dx,
                                      from_queue ? in.dy : rec.dy, from_queue ? in.dz : rec.dz,
                                      from_queue ? in.e : rec.e};
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            ph.pos[a] = src[a][r];
            ph.dir[a] = src[3 + a][r];
          }
          set_energy(s, ph, src[6][r]);
          const uint32_t rp = (from_queue ? in.rng_pos : rec.rng_pos)[r];
          S.rng = (from_queue ? in.rng_buf : rec.rng_buf)[r];
          e.x = rp >> 3;
          idx = (int)(rp & 7u);
          e.y = h;
          ph.exclude = -1;
          if (from_queue) {
            const uint32_t m = in.meta[h];
            e.y = (uint32_t)(in.hid[h] - args.h_begin);
            ph.steps = (int)(m & kMetaSteps);
            ph.exclude = (int)((m >> kMetaExcl) & 7u) - 1;
            x.x = (m >> kMetaEv) & 1u;
            x.y = h;
          } else {
            ph.steps = (int)((f >> 2) & 1u);
          }
          e.w = (uint32_t)run_of(s, args.h_begin + e.y);
          ph.t_exit = R<real>(0);
          aim = (f & 3u) == kRecInImage;
          dest = aim ? kQFly : kQWorld;
          if ((f & 3u) == kRecPendingWorld) {
            smat = s.world_mat;
            dest = kQInteract;
          }
        }
      } else {
        slot_load(S, e, ph, cw, idx);
        ph.exclude = (int)((e.z >> kSlExcl) & 3u) - 1;
        sec.has = (int)((e.z >> kSlSec) & 1u);
        dest = kQFly;
        aim = event == kQFly && ph.t_exit < R<real>(0);
      }
      ph.run = (int)e.w;
      ph.in_head = 0;
      sec.tid = (int)(slot0 + (uint32_t)k);
      hid = args.h_begin + e.y;
      const uint32_t h0 = (uint32_t)hid, h1 = (uint32_t)(hid >> 32);
      if (event == kQInteract) {
        pmat = (int)(cw >> 16);
        pscored = (int)((e.z >> kSlImage) & 1u);
        pv = real_bits(ph.t_exit);
        EventRng g{buf, ahead[threadIdx.x], k0, k1, 0u, h0, h1, e.x, idx};
        g.begin();
        real ed;
        const bool done = pool_interact(s, ph, g, &bc, sec, pmat, (e.z >> kSlRetry) != 0u, trials, kind, ed);
        g.end();
        e.x = g.blk;
        idx = g.idx;
        if (!done) {
          dest = kQInteract;
          smat = pmat;
        } else {
          aim = pscored && ph.alive;
          if (!pscored) {
            dest = kQWorld;
            ph.exclude = -1;
          }
          if constexpr (SPLIT) {
            if (kind == kCompton && s.ss_nc > 0) {
              if ((int)++x.w > s.ss_max) ph.alive = 0;
              else copies = s.ss_nc;
            } else if (kind == kRayleigh) {
              copies = s.ss_nr;
            }
            aim = aim && ph.alive;
          }
          if (!ph.alive) dest = kQRefill;
        }
      }
      if (aim) ph.t_exit = exit_distance(ph.pos, ph.dir, s.bmin, s.bmax);
      if (event == kQWorld || dest == kQFly) {
        // ---- a flight
        if (++ph.steps > kStepCap) {
          atomicAdd(&bc.loop_capped, 1u);
          dest = kQRefill;
        } else {
          TwoWords g;
          g.draw(buf, e.x, idx, 0u, h0, h1, k0, k1);
          if (event == kQWorld) {
            ++n_world;
            ph.in_image = 0;
            if (spect_world_flight(s, ph, g)) {
              smat = s.world_mat;
              pscored = 0;
              dest = kQInteract;
            } else if (ph.alive && ph.in_image) {
              ph.t_exit = R<real>(-1);
              dest = kQFly;
            } else {
              // stopped by a shield, out of the world, or at a head (split copies only are detected there)
              leave = !SPLIT && ph.alive;
              dest = kQRefill;
              if (!leave) ++n_esc;
            }
          } else {
            ph.in_image = 1;
            const int r = image_flight(s, ph, g, smat, pv, pscored, n_wood, n_real);
            dest = r == kInteract ? kQInteract : (ph.in_image ? kQFly : kQWorld);
          }
          g.end(buf, e.x, idx);
        }
      }
    }
    // ---- collective claims: split requests, head-queue entries
    if constexpr (SPLIT) {
      if (event == kQInteract) {
        const bool req_c = copies > 0 && kind == kCompton, req_r = copies > 0 && kind == kRayleigh;
        const size_t kc = queue_claim(q.split_n, req_c, lane, lt_mask);
        const size_t kr = queue_claim(q.split_n + 1, req_r, lane, lt_mask);
        if (copies > 0) {
          // past the capacity the split kernel skips the whole buffer and the pass is repeated
          if (req_c ? kc < q.split_cap : kr < q.split_cap) {
            const size_t j = req_c ? kc : q.split_cap - 1 - kr;
            const SplitQueue<real> sq = SplitQueue<real>::carve(q.split_q, q.split_cap);
            const Real4<real> a = slots[k].a, b = slots[k].b;  // the photon before the interaction
            sq.hid[j] = hid;
            sq.px[j] = a.x;
            sq.py[j] = a.y;
            sq.pz[j] = a.z;
            sq.dx[j] = b.x;
            sq.dy[j] = b.y;
            sq.dz[j] = b.z;
            sq.e[j] = b.w;
            sq.w[j] = s.s_fd_w;
            sq.base[j] = x.z;
            sq.comp[j] = s.mat_comp[pmat];
            sq.run[j] = ph.run;
          }
          x.z += (uint32_t)copies;
        }
      }
    } else {
      if (event == kQWorld) {
        const size_t j = queue_claim(q.out_n, leave, lane, lt_mask);
        if (leave) {
          if (j < q.q_cap) {
            Rng g;
            rng_resume(g, args.seed, hid, (e.x << 3) | (uint32_t)idx, slots[k].rng);
            real v[kEvSlots];
            if (x.x) load_event(in, x.y, v);
            queue_put<real, false>(out, j, ph, g, hid, v, x.x != 0u);
          } else {
            atomicOr(args.status, kStatusQueueOverflow);
          }
          x.x = 0u;  // nothing to score here
        }
      }
    }
    if (k >= 0) {
      PhantomSlot<real> &S = slots[k];
      if (dest == kQRefill && sec.has && !leave) {
        take_secondary(s, ph, sec);
        ph.t_exit = R<real>(-1);
        dest = ph.in_image ? kQFly : kQWorld;
        fresh = true;
        x.w = 0u;
      }
      // ---- the photon back into its slot
      const bool pend = dest == kQInteract;
      if (live) {
        slot_store(S, ph, pend, fresh, smat, pv, trials);
        e.z = (uint32_t)ph.steps | ((uint32_t)idx << kSlIdx) | ((uint32_t)(ph.exclude + 1) << kSlExcl) |
              ((uint32_t)sec.has << kSlSec);
        if (pend) e.z |= (pscored ? 1u << kSlImage : 0u) | (trials ? 1u << kSlRetry : 0u);
      }
      S.e = e;
      if (fresh || leave) S.x.v = x;
    }
    if (event == kQRefill) claims.advance(n);
    Q.put(dest, k, lane, lt_mask);
  }
  stage_counters(args.counters, bc, lane, n_wood, n_real, n_world, 0u, n_singles);
  unsigned long long esc = n_esc;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) esc += __shfl_down_sync(0xffffffffu, esc, o);
  if (lane == 0 && esc) atomicAdd(&args.counters[GG_CNT_ESCAPED], esc);
}

// Phantom stage of primary free flight: the checks of every primary's flight
// (cutoffs, angle, the head its line enters); the optical depth of those that
// pass is walked by k_spect_walk.  One record per thread, nothing to batch.
template <typename real>
__global__ void __launch_bounds__(256) k_spect_primary(Scene<real> s, KernelArgs args, StageArgs q) {
  __shared__ BlockCounters bc;
  if (threadIdx.x == 0) bc = BlockCounters{0, 0, 0, 0, 0, 0, 0, 0};
  __syncthreads();
  const Records<real> rec = Records<real>::carve(args.records, args.rec_cap);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const uint64_t n = args.h_end - args.h_begin;
  const unsigned lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  unsigned int n_world = 0, n_esc = 0;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t h = i0 + threadIdx.x, hid = args.h_begin + h, r = hid - args.rec_first;
    Photon<real> ph;
    bool push = false;
    uint32_t f = kRecDead;
    if (h < n) f = rec.flags[r];
    if ((f & 3u) != kRecDead) {
      ph.pos[0] = rec.px[r];
      ph.pos[1] = rec.py[r];
      ph.pos[2] = rec.pz[r];
      ph.dir[0] = rec.dx[r];
      ph.dir[1] = rec.dy[r];
      ph.dir[2] = rec.dz[r];
      ph.e = rec.e[r];
      ph.steps = (int)((f >> 2) & 1u) + 1;  // (one flight: far below the step cap)
      ph.alive = 1;
      ph.exclude = -1;
      ph.head = ph.hreg = 0;
      ph.w = s.s_fd_w;  // 1, or the forced direction's cone weight
      ph.run = run_of(s, hid);
      ++n_world;
      real tb;
      push = ff_target(s, ph, s.ss_cos, tb) != 0;
      if (!push) ++n_esc;
    }
    const size_t k = queue_claim(q.out_n, push, lane, lt_mask);
    if (push) {
      if (k < q.q_cap) {
        Rng g;
        rng_resume(g, args.seed, hid, rec.rng_pos[r], rec.rng_buf[r]);
        real v[kEvSlots];
        queue_put<real, true>(out, k, ph, g, hid, v, false);
      } else {
        atomicOr(args.status, kStatusQueueOverflow);
      }
    }
  }
  if (n_esc) atomicAdd(&bc.escaped, n_esc);
  stage_counters(args.counters, bc, lane, 0u, 0u, n_world, 0u, 0u);
}

// Head stage.  Input: the head queue; output: the return queue.  Each lane
// carries its photon's event in registers and scores it when the photon
// dies.
template <typename real, int MINB, bool FF>
__global__ void __launch_bounds__(256, MINB) k_spect_head(Scene<real> sg, KernelArgs args, StageArgs q) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  __shared__ real sec_store[6 * 256];
  Scene<real> s = sg;
  stage_tables(sg, s, smem_raw, bc);
  const PQueue<real> in = PQueue<real>::carve(q.in_q, q.q_cap);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const uint64_t n_items = min((uint64_t)*q.in_n, (uint64_t)q.q_cap);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  __shared__ uint64_t wpool[kBlock / 32][2];  // per warp: claimed histories not yet handed out
  uint64_t *pool = wpool[threadIdx.x >> 5];
  if (lane == 0) pool[0] = pool[1] = 0;
  __syncwarp();

  Photon<real> ph;
  ph.alive = 0;
  ph.run = 0;
  Secondary<real> sec;
  sec.base = sec_store;
  sec.stride = blockDim.x;
  sec.tid = threadIdx.x;
  sec.has = 0;
  Event<real> ev;
  ev.clear();
  Rng g;
  int state = kRefill;
  bool in_hist = false;
  int pmat = 0, pscored = 0;
  unsigned int n_world = 0, n_head = 0, n_singles = 0;

  for (;;) {
    // phase chosen per block: all warps run the same code region at the same
    // time (instruction-cache locality); thresholds are per warp
    const unsigned m_ref = __ballot_sync(0xffffffffu, state == kRefill);
    const int c_ref = __syncthreads_count(state == kRefill);
    const int c_fly = __syncthreads_count(state == kFly);
    const int c_int = __syncthreads_count(state == kInteract);
    if (c_ref + c_fly + c_int == 0) break;
    const int n_warps = (int)(blockDim.x >> 5);
    int phase;
    if (c_ref >= args.refill_min * n_warps || (c_fly + c_int) == 0) phase = kRefill;
    else if (c_int >= args.interact_min * n_warps || c_fly == 0) phase = kInteract;
    else phase = kFly;

    if (phase == kRefill) {
      const bool need = state == kRefill;
      if (need && in_hist) {
        n_singles += score_singles(s, ev, ph.run, g);
        in_hist = false;
      }
      const uint64_t h = warp_pool_claim(pool, m_ref, lane, lt_mask, args.next, args.chunk);
      if (need) {
        if (h >= n_items) {
          state = kDone;
        } else {
          bool has_ev;
          queue_get<real, FF>(s, in, h, ph, g, args.seed, has_ev);
          if (has_ev) {
            real v[kEvSlots];
            load_event(in, h, v);
            event_from(v, ev);
          } else {
            ev.clear();
          }
          ph.in_head = 1;
          ph.in_image = 0;
          state = kFly;
          in_hist = true;
        }
      }
    } else if (phase == kInteract) {
      if (state == kInteract) {
        state = head_interaction(s, ph, g, &bc, pmat, pscored, sec, ev);
        if (state == kRefill && sec.has) {
          pop_secondary(s, ph, sec);
          state = kFly;
        }
      }
    } else {
      if (state == kFly) {
        state = head_stage_flight<real, FF>(s, ph, g, &bc, pmat, pscored, n_world, n_head);
        if (state == kRefill && sec.has) {
          pop_secondary(s, ph, sec);
          state = kFly;
        }
      }
      const bool push = state == kPush;
      const size_t k = queue_claim(q.out_n, push, lane, lt_mask);
      if (push) {
        if (k < q.q_cap) {
          real v[kEvSlots];
          event_to(ev, v);
          queue_put<real, FF>(out, k, ph, g, rng_history(g), v, true);
        } else {
          atomicOr(args.status, kStatusQueueOverflow);
        }
        in_hist = false;
        state = kRefill;
      }
    }
  }
  stage_counters(args.counters, bc, lane, 0u, 0u, n_world, n_head, n_singles);
}

// A projection tally as FP64 values, for its copy to the caller: counts, fixed
// point weights (2^-32), or their squares (low 32 bits, rest; the sum of two
// exact products, rounded once).  Bound by memory: 16 or 24 bytes per pixel.
// The conversion on the host cost 25 to 30 ns per pixel (pageable copy, a loop,
// fresh pages): 2 heads x 120 positions x 3 windows x 128 x 128, weights and
// squares, 36 ms.
template <int KIND>
__global__ void __launch_bounds__(256) k_projection_f64(const unsigned long long *src, double *dst, size_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    double v;
    if constexpr (KIND == kProjSquares) {
      const ulonglong2 b = reinterpret_cast<const ulonglong2 *>(src)[i];
      const double lo = (double)b.x * 5.421010862427522e-20;  // 2^-64
      const double hi = (double)b.y * 2.3283064365386963e-10;  // 2^-32
      v = hi + lo;
    } else {
      v = (double)src[i];
      if constexpr (KIND == kProjWeights) v = v * 2.3283064365386963e-10;
    }
    dst[i] = v;
  }
}

cudaError_t launch_projection_f64(int kind, const unsigned long long *src, double *dst, size_t n, int n_sm,
                                  cudaStream_t st) {
  const int grid = n_sm * 8;
  if (kind == kProjCounts) k_projection_f64<kProjCounts><<<grid, 256, 0, st>>>(src, dst, n);
  else if (kind == kProjWeights) k_projection_f64<kProjWeights><<<grid, 256, 0, st>>>(src, dst, n);
  else if (kind == kProjSquares) k_projection_f64<kProjSquares><<<grid, 256, 0, st>>>(src, dst, n);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

template <typename real, int MINB, bool FF>
static cudaError_t launch_head_v(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int grid, int block,
                                 size_t smem, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_spect_head<real, MINB, FF>, 200 * 1024, configured);
  if (e != cudaSuccess) return e;
  k_spect_head<real, MINB, FF><<<grid, block, smem, st>>>(s, a, q);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_spect_head(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int grid, int block,
                              size_t smem, int minb, cudaStream_t st) {
  // free flight: one register budget (4 blocks of 256 threads per SM); a
  // smaller grid computed for another budget is a valid launch of it
  if (s.ff) return launch_head_v<real, 4, true>(s, a, q, grid, block, smem, st);
  if (minb <= 2) return launch_head_v<real, 2, false>(s, a, q, grid, block, smem, st);
  if (minb == 3) return launch_head_v<real, 3, false>(s, a, q, grid, block, smem, st);
  return launch_head_v<real, 4, false>(s, a, q, grid, block, smem, st);
}

template <typename real, bool SPLIT>
static cudaError_t launch_phantom_v(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, const PoolPlan &p,
                                    cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_spect_phantom<real, SPLIT>, 227 * 1024, configured);
  if (e != cudaSuccess) return e;
  k_spect_phantom<real, SPLIT><<<p.grid, p.block, p.smem, st>>>(s, a, q, p.slots, p.gang_threads);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_spect_phantom(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, const PoolPlan &p,
                                 int n_sm, cudaStream_t st) {
  if (s.ff == kFfPrimary) {
    k_spect_primary<real><<<n_sm * 8, 256, 0, st>>>(s, a, q);
    return cudaGetLastError();
  }
  return s.ff == kFfScatter ? launch_phantom_v<real, true>(s, a, q, p, st) : launch_phantom_v<real, false>(s, a, q, p, st);
}

template <typename real>
size_t phantom_slot_bytes() {
  return sizeof(PhantomSlot<real>);
}

template <typename real>
cudaError_t spect_head_occupancy(int block, size_t smem, int minb, int *bps) {
  if (minb <= 2) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_spect_head<real, 2, false>, block, smem);
  if (minb == 3) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_spect_head<real, 3, false>, block, smem);
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_spect_head<real, 4, false>, block, smem);
}

template <typename real>
cudaError_t launch_spect_split(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int n_sm,
                               cudaStream_t st) {
  int bps = 1;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_spect_split<real>, kBlock, 0);
  if (e != cudaSuccess) return e;
  if (bps < 1) bps = 1;
  k_spect_split<real><<<n_sm * bps, kBlock, 0, st>>>(s, a, q);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_spect_walk(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int block, size_t smem,
                              int n_sm, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_spect_walk<real>, 200 * 1024, configured);
  int bps = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_spect_walk<real>, block, smem);
  if (e != cudaSuccess) return e;
  if (bps < 1) bps = 1;
  k_spect_walk<real><<<n_sm * bps, block, smem, st>>>(s, a, q);
  return cudaGetLastError();
}

template cudaError_t launch_spect_walk<float>(const Scene<float> &, const KernelArgs &, const StageArgs &, int,
                                              size_t, int, cudaStream_t);
template cudaError_t launch_spect_walk<double>(const Scene<double> &, const KernelArgs &, const StageArgs &, int,
                                               size_t, int, cudaStream_t);
template size_t split_bytes<float>(size_t);
template size_t split_bytes<double>(size_t);
template cudaError_t launch_spect_split<float>(const Scene<float> &, const KernelArgs &, const StageArgs &, int,
                                               cudaStream_t);
template cudaError_t launch_spect_split<double>(const Scene<double> &, const KernelArgs &, const StageArgs &, int,
                                                cudaStream_t);
template size_t queue_bytes<float>(size_t);
template size_t queue_bytes<double>(size_t);
template size_t phantom_slot_bytes<float>();
template size_t phantom_slot_bytes<double>();
template cudaError_t launch_spect_phantom<float>(const Scene<float> &, const KernelArgs &, const StageArgs &,
                                                 const PoolPlan &, int, cudaStream_t);
template cudaError_t launch_spect_phantom<double>(const Scene<double> &, const KernelArgs &, const StageArgs &,
                                                  const PoolPlan &, int, cudaStream_t);
template cudaError_t launch_spect_head<float>(const Scene<float> &, const KernelArgs &, const StageArgs &, int, int,
                                              size_t, int, cudaStream_t);
template cudaError_t launch_spect_head<double>(const Scene<double> &, const KernelArgs &, const StageArgs &, int, int,
                                               size_t, int, cudaStream_t);
template cudaError_t spect_head_occupancy<float>(int, size_t, int, int *);
template cudaError_t spect_head_occupancy<double>(int, size_t, int, int *);

}  // namespace gg
