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

// Whether a photon of direction d scattered by theta (cos, sin^2) can pass the
// angle check of some head (ff_target): over the azimuth, the largest cosine
// between the new direction and a head axis u is cos(theta - theta_u) =
// cos(theta) (d.u) + sin(theta) sqrt(1 - (d.u)^2).  A margin of 1e-4 on the
// cosine keeps every direction the full check would accept (rounding is far
// below it), so dropping the others changes no result.
template <typename real>
__device__ __forceinline__ bool cone_reachable(const Scene<real> &s, int run, const real d[3], real cost, real sint2,
                                               real cos_min) {
  const real sint = gg_sqrt(sint2 > R<real>(0) ? sint2 : R<real>(0));
  const real lim = cos_min - R<real>(1e-4);
  for (int h = 0; h < s.n_heads; ++h) {
    const HeadFrame<real> f = head_frame(s, run, h);
    const real c0 = dot3(d, f.u);
    real s0 = R<real>(1) - c0 * c0;
    s0 = gg_sqrt(s0 > R<real>(0) ? s0 : R<real>(0));
    real m = cost * c0;
    m = m + sint * s0;
    if (!(m < lim)) return true;
  }
  return false;
}

// Copies of one warp that passed the scattering-angle test and wait for the
// rest of their scattering and the head checks, kSplitPend at most: the copy
// index, the sampled (eps, 1 - cos, sin^2) of a Compton or (cos, -, -) of a
// Rayleigh scattering, and the words of the copy's stream drawn so far.
constexpr int kSplitPend = 64;
template <typename real>
struct SplitPending {
  uint64_t i[kSplitPend];
  real a[kSplitPend], b[kSplitPend], c[kSplitPend];
  uint32_t words[kSplitPend];
};

// Scatter splitting, the copies (GateScatterSplittingFreeFlightOptn.cpp:69-149):
// one thread per copy.  Request r of the phantom stage holds the photon
// before a Compton (or Rayleigh) interaction; its copy c re-samples that
// interaction from there on Philox stream 2 + base + c of the history, with
// 1 / n of the weight, and flies freely to a head: the intersection check of
// the angular acceptance is the flight itself (a copy that misses every head
// cannot be detected), the angle check comes before the optical depth.
// A copy whose line enters a head (past the checks) goes to the walk queue
// (q.out_q), where k_spect_walk computes its optical depth: the few copies
// that pass then walk the voxels with full warps.  Compton requests fill the
// buffer from the front and Rayleigh requests from the back; when together
// they overflowed it, nothing is done (the host repeats the pass on fewer
// histories).
// Most copies scatter away from every head: right after the rejection loop
// the scattering angle alone decides that (cone_reachable), and only the
// others draw their azimuth and meet the full check.  Those wait in a
// per-warp buffer until 32 of them fill the warp's lanes, so the azimuth,
// the rotation and the head checks run on full warps; each copy's arithmetic
// and draws are those of the plain sequence.
template <typename real>
__global__ void __launch_bounds__(256) k_spect_split(Scene<real> sg, KernelArgs args, StageArgs q) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  __shared__ SplitPending<real> pend_all[kBlock / 32];
  Scene<real> s = sg;
  stage_tables(sg, s, smem_raw, bc);
  const uint64_t n_c = *q.split_n, n_r = q.split_n[1];
  if (n_c + n_r > (uint64_t)q.split_cap) return;
  const uint64_t per_c = (uint64_t)s.ss_nc, per_r = (uint64_t)s.ss_nr;
  const uint64_t all_c = n_c * per_c, total = all_c + n_r * per_r;
  const SplitQueue<real> sq = SplitQueue<real>::carve(q.split_q, q.split_cap);
  const PQueue<real> out = PQueue<real>::carve(q.out_q, q.q_cap);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  SplitPending<real> &P = pend_all[threadIdx.x >> 5];
  int np = 0;  // copies waiting in P (the same in every lane of the warp)
  unsigned int n_world = 0;
  // copy i: its request, the photon before the interaction, its stream
  auto load_copy = [&](uint64_t i, Photon<real> &cp, Rng &gc, uint64_t &hid) {
    uint64_t r;
    uint32_t c, n;
    if (i < all_c) {
      r = i / per_c;
      c = (uint32_t)(i - r * per_c);
      n = (uint32_t)per_c;
    } else {
      const uint64_t j = i - all_c, rr = j / per_r;
      c = (uint32_t)(j - rr * per_r);
      r = (uint64_t)q.split_cap - 1 - rr;
      n = (uint32_t)per_r;
    }
    hid = sq.hid[r];
    cp.pos[0] = sq.px[r];
    cp.pos[1] = sq.py[r];
    cp.pos[2] = sq.pz[r];
    cp.dir[0] = sq.dx[r];
    cp.dir[1] = sq.dy[r];
    cp.dir[2] = sq.dz[r];
    cp.e = sq.e[r];  // the energy-grid state only where a sampling uses it (set_energy)
    cp.w = sq.w[r] / (real)n;
    cp.alive = 1;
    cp.run = sq.run[r];
    gc.init(args.seed, hid, 2u + sq.base[r] + c);
    return r;
  };
  // the waiting copies P[k0 + lane] (lane < cnt): the rest of the scattering,
  // the head checks, and the walk queue (every lane of the warp calls it)
  auto finish = [&](int k0, int cnt) {
    Photon<real> cp;
    Rng gc;
    uint64_t hid = 0;
    bool push = false;
    if ((int)lane < cnt) {
      const int k = k0 + (int)lane;
      const uint64_t i = P.i[k];
      load_copy(i, cp, gc, hid);
      // the stream after its first `w` words: the state an Rng reaches by drawing them
      const uint32_t w = P.words[k];
      if ((w & 3u) == 0u) {
        gc.blk = w >> 2;
        gc.idx = 4;
      } else {
        const uint4 b = philox_block(w >> 2, gc.stream, gc.h0, gc.h1, gc.k0, gc.k1);
        gc.buf[0] = b.x;
        gc.buf[1] = b.y;
        gc.buf[2] = b.z;
        gc.buf[3] = b.w;
        gc.blk = (w >> 2) + 1u;
        gc.idx = (int)(w & 3u);
      }
      if (i < all_c) compton_finish(s, cp, gc, P.a[k], P.b[k], P.c[k]);
      else rayleigh_finish(cp, gc, P.a[k]);
      if (cp.alive) {
        cp.exclude = -1;
        cp.steps = 0;
        cp.head = 0;
        cp.hreg = 0;
        ++n_world;
        real tb;
        push = ff_target(s, cp, s.ss_cos, tb) != 0;  // with the angle check of the angular acceptance
        if (!push) atomicAdd(&bc.escaped, 1u);
      }
    }
    const size_t kq = queue_claim(q.out_n, push, lane, lt_mask);
    if (push && kq < q.q_cap) {
      real v[kEvSlots];
      queue_put<real, true>(out, kq, cp, gc, hid, v, false);
    }
  };
  // the loop bound is the same for all threads of a block: queue claims stay warp-collective
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < total; i0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = i0 + threadIdx.x;
    bool wait = false;
    real a = R<real>(0), b = R<real>(0), c = R<real>(0);
    Rng gc;
    if (i < total) {
      Photon<real> cp;
      uint64_t hid;
      const uint64_t r = load_copy(i, cp, gc, hid);
      bool dead = false, out_of_cone;
      if (i < all_c) {
        compton_kn(cp.e, gc, &bc, a, b, c);
        // (below the energy cut the copy dies in compton_finish)
        dead = a * cp.e < s.e_min;
        out_of_cone = !dead && s.ss_cos > R<real>(-1) && !cone_reachable(s, cp.run, cp.dir, R<real>(1) - b, c, s.ss_cos);
      } else {
        set_energy(s, cp, cp.e);
        a = rayleigh_cost(s, sq.comp[r], cp, gc, &bc);
        out_of_cone = s.ss_cos > R<real>(-1) && !cone_reachable(s, cp.run, cp.dir, a, rayleigh_sint2(a), s.ss_cos);
      }
      if (out_of_cone) {  // a live copy that fails the head checks, as counted there
        ++n_world;
        atomicAdd(&bc.escaped, 1u);
      }
      wait = !dead && !out_of_cone;
    }
    const unsigned m = __ballot_sync(0xffffffffu, wait);
    if (wait) {
      const int k = np + __popc(m & lt_mask);
      P.i[k] = i;
      P.a[k] = a;
      P.b[k] = b;
      P.c[k] = c;
      P.words[k] = (gc.blk - 1u) * 4u + (uint32_t)gc.idx;  // (the loops drew at least one word)
    }
    np += __popc(m);
    __syncwarp();
    if (np >= 32) {
      finish(np - 32, 32);
      np -= 32;
      __syncwarp();
    }
  }
  if (np > 0) finish(0, np);
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
template <typename real, bool SPLIT>
__global__ void __launch_bounds__(PoolShape<real>::kBlock, 1)
    k_spect_phantom(const __grid_constant__ Scene<real> sg, KernelArgs args, StageArgs q, int n_slots) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  using Shape = PoolShape<real>;
  constexpr int kGangs = Shape::kBlock / (32 * Shape::kGang), kGang = 32 * Shape::kGang;
  __shared__ __align__(16) unsigned push[kGangs][3 * kQueues];
  __shared__ __align__(16) uint32_t ahead[Shape::kBlock][4];  // EventRng's second block of each thread
  __shared__ uint16_t ring[kGangs][kQueues * Shape::kRing];
  __shared__ unsigned long long s_claim[kGangs];
  Scene<real> s = sg;
  const unsigned lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  const int gang = (int)threadIdx.x / kGang, gang0 = gang * kGang;
  const int gangs = ((int)blockDim.x + kGang - 1) / kGang;
  // dynamic shared memory: slots of the gangs, tables
  PhantomSlot<real> *const slots = reinterpret_cast<PhantomSlot<real> *>(smem_raw) + gang * n_slots;
  EventQueues<Shape::kRing> Q;
  Q.init(gang, threadIdx.x - (unsigned)gang0, min((unsigned)kGang, blockDim.x - (unsigned)gang0), ring[gang], push[gang],
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
  HistList<real> l{nullptr, nullptr, 0, 0};  // never scored here
  Tally<real> t{nullptr, nullptr};
  Event<real> ev;
  ev.clear();
  Rng g;
  int state = kRefill;
  bool in_hist = false;
  int pmat = 0, pscored = 0;
  uint32_t pv = 0;
  unsigned int n_dep = 0, n_world = 0, n_head = 0, n_singles = 0;

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
        state = do_interaction<real, true>(s, ph, g, &bc, pmat, pv, pscored, l, t, sec, n_dep, ev);
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
  k_spect_phantom<real, SPLIT><<<p.grid, p.block, p.smem, st>>>(s, a, q, p.slots);
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
cudaError_t launch_spect_split(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int block, size_t smem,
                               int n_sm, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_spect_split<real>, 200 * 1024, configured);
  int bps = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_spect_split<real>, block, smem);
  if (e != cudaSuccess) return e;
  if (bps < 1) bps = 1;
  k_spect_split<real><<<n_sm * bps, block, smem, st>>>(s, a, q);
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
                                               size_t, int, cudaStream_t);
template cudaError_t launch_spect_split<double>(const Scene<double> &, const KernelArgs &, const StageArgs &, int,
                                                size_t, int, cudaStream_t);
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
