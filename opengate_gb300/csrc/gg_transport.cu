// gg_transport.cu - photon transport through a voxelised image with DoseActor scoring.
//
// Replaces, for photons in a voxelised volume, Geant4's stepping through the
// replica/parameterised voxels of ImageVolume
// (opengate/geometry/volumes.py:1093-1125, GateImageNestedParameterisation.cpp:47-75)
// and the scoring of GateDoseActor::SteppingAction / ScoreSquaredValue /
// FlushSquaredValues (core/opengate_core/opengate_lib/GateDoseActor.cpp:180-243, 359-397).
//
// Kernel design (one GB300, one process):
//   * a source stage samples the primaries into coalesced records;
//   * the transport stage keeps more photons than threads in shared memory and
//     runs one kind of event at a time on full warps (gg_pool.cuh); only the
//     track-length estimator still carries one photon per thread;
//   * Woodcock (delta) tracking against a per-energy majorant inside the image
//     box; analytic free flight in the world material outside it;
//   * the majorant, total attenuation rows and the label->(composition,
//     density) table are staged in shared memory; labels are read through the
//     read-only path (the image is L2-resident up to ~60 M voxels);
//   * every history keeps its deposits in a list of (voxel, sum); when the
//     history ends each entry adds q = round(sum * 2^32) to the edep tally
//     (64-bit integer atomic) and q^2 to a 128-bit edep-squared tally: the
//     history-by-history squared sum of GateDoseActor, order independent and
//     therefore bit-reproducible;
//   * a third kernel flushes the per-batch fixed-point tallies into the
//     float64 images (and clears them), one voxel per thread, coalesced.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gg_device.cuh"
#include "gg_internal.h"
#include "gg_physics.cuh"
#include "gg_pool.cuh"
#include "gg_queue.cuh"
#include "gg_spect.cuh"

namespace gg {

// First step of a sampled primary in the source stage: a photon outside the
// image takes its first world flight here (dose; SPECT leaves it to the
// transport stage, whose world step also targets the heads).  Sets the
// record state; true when a world step was taken.
template <typename real>
__device__ __forceinline__ bool first_flight(const Scene<real> &s, RngAhead &g, Photon<real> &ph, uint32_t &state,
                                             uint32_t &steps, BlockCounters *bc) {
  if (ph.in_image) {
    state = kRecInImage;
    return false;
  }
  if (s.spect) {
    state = kRecWorld;
    return false;
  }
  steps = 1;
  real inf = gg_inf(real(0));
  real tin = ph.can_enter ? entry_distance(ph.pos, ph.dir, s.bmin, s.bmax) : inf;
  real wlo[3] = {-s.whalf[0], -s.whalf[1], -s.whalf[2]};
  real tout = exit_distance(ph.pos, ph.dir, wlo, s.whalf);
  int wm = s.world_mat;
  real mu = interp_row(s.sig + (size_t)s.mat_comp[wm] * s.n_e, ph.ei);
  mu = s.mat_rho[wm] * mu;
  real u = u01_open0<real>(g);
  real sd = -gg_log(u);
  sd = sd / mu;
  if (sd < tin && sd < tout) {
#pragma unroll
    for (int k = 0; k < 3; ++k) ph.pos[k] = ph.pos[k] + sd * ph.dir[k];
    state = kRecPendingWorld;
  } else if (tin <= tout) {
#pragma unroll
    for (int k = 0; k < 3; ++k) ph.pos[k] = ph.pos[k] + tin * ph.dir[k];
    state = kRecInImage;
  } else {
    atomicAdd(&bc->escaped, 1u);
  }
  return true;
}

template <typename real>
__device__ __forceinline__ void write_record(const Records<real> &rec, uint64_t i, const Photon<real> &ph,
                                             const RngAhead &g, uint32_t state, uint32_t steps, uint32_t sim) {
  rec.px[i] = ph.pos[0];
  rec.py[i] = ph.pos[1];
  rec.pz[i] = ph.pos[2];
  rec.dx[i] = ph.dir[0];
  rec.dy[i] = ph.dir[1];
  rec.dz[i] = ph.dir[2];
  rec.e[i] = ph.e;
  rec.flags[i] = state | (steps << 2);
  rec.rng_pos[i] = (g.blk << 3) | (uint32_t)g.idx;
  rec.rng_buf[i] = make_uint4(g.buf[0], g.buf[1], g.buf[2], g.buf[3]);
  rec.sim[i] = sim;
}

// Source stage: one thread per history.  Samples the primary
// (GateGenericSource::GeneratePrimaries order), places it, and performs the
// first transport iteration when the photon starts in the world (free flight
// to the image, to an air interaction, or out of the world).
// MULTI: batched simulations (Scene::sims): the thread's history picks its
// simulation, whose geometry, source and Philox key it then uses.  Without
// MULTI, isotropic directions with an acceptance loop are sampled by the
// warp together (warp_iso_direction_accepted).
template <typename real, bool MULTI>
__global__ void __launch_bounds__(256) k_generate(Scene<real> s, KernelArgs a) {
  __shared__ BlockCounters bc;
  if (threadIdx.x == 0) bc = BlockCounters{0, 0, 0, 0, 0, 0, 0, 0};
  __syncthreads();
  const uint64_t n = a.h_end - a.h_begin;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool sampled = false, world_step = false;  // counted per block below
  // isotropic directions with an acceptance loop: the warp samples them together
  const bool warp_dirs = !MULTI && s.dir_type == GG_DIR_ISO && s.n_accept > 0;
  if (warp_dirs) {
    Records<real> rec = Records<real>::carve(a.records, a.rec_cap);
    RngAhead g;  // blocks made on demand: the warp's trials read the stream directly
    g.init(a.seed, a.h_begin + i, 0u);
    g.ahead = false;
    Photon<real> ph;
    const bool live = i < n;
    if (live) sample_position(s, g, ph, &bc);
    int st = warp_iso_direction_accepted(s, g, ph, live, &bc);
    if (live) {
      uint32_t state = kRecDead, steps = 0;
      if (st != GG_OK) {
        atomicOr(a.status, (unsigned int)st);
      } else {
        sample_energy(s, g, ph);
        sampled = true;
        start_photon(s, ph);
        world_step = first_flight(s, g, ph, state, steps, &bc);
      }
      write_record(rec, i, ph, g, state, steps, 0u);
    }
  } else if (i < n) {
    Records<real> rec = Records<real>::carve(a.records, a.rec_cap);
    RngAhead g;
    uint32_t sim = 0;
    if constexpr (MULTI) {
      const uint64_t h = a.h_begin + i;
      sim = (uint32_t)find_sim(s.sims, s.n_sims, h);
      const SimDesc<real> &d = s.sims[sim];
      bind_geometry(s, d, s.labels, s.sim_maj + (size_t)sim * s.n_e);
      bind_source(s, d);
      g.start(d.seed, h - d.h_begin, 0u);
    } else {
      g.start(a.seed, a.h_begin + i, 0u);
    }
    Photon<real> ph;
    if (s.dir_type == GG_DIR_FORCED) {  // the head (and run) the history's photon is aimed at
      const uint64_t h = a.h_begin + i;
      ph.run = s.run_base + (int)((h - s.run_first) / s.run_len);
      ph.head = (int)(h % (uint64_t)s.n_heads);
    }
    uint32_t state = kRecDead, steps = 0;
    int st = sample_primary(s, g, ph, &bc);
    if (st != GG_OK) {
      atomicOr(a.status, (unsigned int)st);
    } else {
      sampled = true;
      start_photon(s, ph);
      world_step = first_flight(s, g, ph, state, steps, &bc);
    }
    write_record(rec, i, ph, g, state, steps, sim);
  }
  const int n_hist = __syncthreads_count(sampled);
  const int n_world = __syncthreads_count(world_step);
  if (threadIdx.x == 0) {
    unsigned long long *cnt = a.counters;
    if (n_hist) atomicAdd(&cnt[GG_CNT_HISTORIES], (unsigned long long)n_hist);
    if (bc.skipped) atomicAdd(&cnt[GG_CNT_SKIPPED], (unsigned long long)bc.skipped);
    if (bc.escaped) atomicAdd(&cnt[GG_CNT_ESCAPED], (unsigned long long)bc.escaped);
    if (bc.loop_capped) atomicAdd(&cnt[GG_CNT_LOOP_CAPPED], (unsigned long long)bc.loop_capped);
    if (n_world) atomicAdd(&cnt[GG_CNT_WORLD_STEPS], (unsigned long long)n_world);
  }
}

// Adds the lanes' counts to a counter (out of line: one copy of the exchange).
static __device__ __noinline__ void warp_count(unsigned long long *counter, unsigned int v) {
  unsigned long long x = v;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if ((threadIdx.x & 31u) == 0u && x) atomicAdd(counter, x);
}

// The dose tally from voxel `off` on (batched simulations: the simulation's part).
template <typename real>
__device__ __forceinline__ Tally<real> tally_at(const KernelArgs &a, size_t off, real) {
  return Tally<real>{a.acc_e + off, a.acc_e2 ? a.acc_e2 + 2 * off : nullptr};
}

// Transport stage: the pooled event loop of gg_pool.cuh.  Events: a new history
// (the ended one's voxel list goes to the tallies first), a Woodcock step in
// the image, a free flight in the world, an interaction; a photon that starts
// or scatters in the image takes its next Woodcock step in the same round.
// The order of operations inside each history, hence its result, does not
// depend on which lane or round executes them.
// Bound by instruction issue and by the gangs' barrier: 256 x 256 x 160 CT, 1e8
// histories to 6 MeV, 47.9 -> 30.4 ms against one photon per thread with block-wide phases
// (203 warp instructions per history at 21.5 active lanes; 379 at 8.6); 24
// batched simulations 22.8 -> 14.1 ms, FP64 9.2 -> 4.2 ms per 1e6.
// MULTI: batched simulations; DG: dose tally on a grid of its own (1: edep,
// 2: edep and dose), Scene::dgrid.
template <typename real, bool MULTI, int DG>
__global__ void __launch_bounds__(PoolShape<real>::kBlock, 1) k_transport_pool(Scene<real> sg, KernelArgs args, int n_slots) {
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
  DoseSlot<real> *const slots = reinterpret_cast<DoseSlot<real> *>(smem_raw) + gang * n_slots;
  EventQueues<Shape::kRing> Q;
  Q.init(gang, threadIdx.x - (unsigned)gang0, min((unsigned)kGang, blockDim.x - (unsigned)gang0), ring[gang], push[gang],
         (unsigned)n_slots);
  for (int i = (int)Q.tid; i < n_slots; i += (int)Q.size) slots[i].e = make_uint4(0u, 0u, 0u, 0u);
  stage_tables(sg, s, smem_raw + sizeof(DoseSlot<real>) * (size_t)(gangs * n_slots), bc);

  const Records<real> rec = Records<real>::carve(args.records, args.rec_cap);
  Tally<real> t{args.acc_e, args.acc_e2};
  const Tally<real> td{args.acc_d, args.acc_d2};
  const uint32_t n_hist = (uint32_t)(args.h_end - args.h_begin);
  const uint32_t slot0 = (blockIdx.x * (uint32_t)gangs + (uint32_t)gang) * (uint32_t)n_slots;
  const uint32_t all_slots = gridDim.x * (uint32_t)(gangs * n_slots);  // global scratch: one column per slot
  Secondary<real> sec;
  sec.base = reinterpret_cast<real *>(args.slot_scratch);
  sec.stride = (int)all_slots;
  GlobalList<real> ld;
  ld.ga = sec.base + 6 * (size_t)all_slots;
  ld.gv = reinterpret_cast<uint32_t *>(ld.ga + kHistList * (size_t)all_slots);
  ld.slots = all_slots;
  unsigned int n_wood = 0, n_real = 0, n_dep = 0, n_world = 0, n_ent = 0, n_over = 0, n_esc = 0;
  ItemClaims claims;
  claims.init();

  for (;;) {
    int k;
    unsigned n;
    const int event = Q.round(k, n);
    if (event == kQNone) break;
    int dest = kQNone;
    if (event == kQRefill) {
      claims.take(Q, n, args.next, args.chunk, n_hist, &s_claim[gang]);
      // the ended histories' voxel lists
      lists_flush(slots, max(k, 0), k >= 0 ? (int)((slots[k].e.z >> kSlList) & 15u) : 0,
                  reinterpret_cast<uint16_t *>(ahead[threadIdx.x & ~31u]), lane,
                  [&](const DoseSlot<real> &S) {
                    if constexpr (MULTI) return tally_at(args, sg.sims[S.e.w].vox_off, real(0));
                    else return t;
                  },
                  n_ent);
    }
    if (k >= 0) {
      DoseSlot<real> &S = slots[k];
      uint4 e = S.e;
      int n_list = (int)((e.z >> kSlList) & 15u);
      if constexpr (DG == 2) {
        ld.at = slot0 + (uint32_t)k;
        ld.n = (int)e.w;
      }
      auto bind = [&](uint32_t sim) {  // batched simulations: the history's geometry, majorant and tally
        const SimDesc<real> &d = sg.sims[sim];
        bind_geometry(s, d, sg.labels, sg.sim_maj + (size_t)sim * sg.n_e);
        t = tally_at(args, d.vox_off, real(0));
      };
      if constexpr (MULTI) bind(e.w);
      Photon<real> ph;
      ph.alive = 1;
      uint32_t cw = 0, pv = 0, trials = 0;
      int pmat = 0, pscored = 0, idx = 0;
      bool fresh = event != kQFly && event != kQWorld;  // direction and energy change
      bool live = true;                                 // the slot holds a photon
      bool aim = false;                                 // its path to the image boundary is not known (in a slot: negative)
      sec.has = 0;
      uint32_t *const buf = &S.rng.x;
      if (event == kQRefill) {
        n_list = 0;
        if constexpr (DG == 2) ld.flush(td);
        uint32_t h, f = kRecDead;
        const bool have = claims.item(Q.tid, h);
        if (have) f = rec.flags[h];
        dest = have || !claims.exhausted ? kQRefill : kQNone;
        live = (f & 3u) != kRecDead;
        e = make_uint4(0u, h, 0u, 0u);
        if (live) {
          if constexpr (MULTI) {
            e.w = rec.sim[h];
            bind(e.w);
          }
          ph.pos[0] = rec.px[h];
          ph.pos[1] = rec.py[h];
          ph.pos[2] = rec.pz[h];
          ph.dir[0] = rec.dx[h];
          ph.dir[1] = rec.dy[h];
          ph.dir[2] = rec.dz[h];
          set_energy(s, ph, rec.e[h]);
          const uint32_t rp = rec.rng_pos[h];
          S.rng = rec.rng_buf[h];
          e.x = rp >> 3;
          idx = (int)(rp & 7u);
          ph.steps = (int)((f >> 2) & 1u);
          ph.can_enter = 1;
          ph.t_exit = R<real>(0);
          if ((f & 3u) == kRecInImage) {
            aim = true;
            dest = kQFly;
          } else if ((f & 3u) == kRecWorld) {
            dest = kQWorld;
          } else {
            pmat = s.world_mat;
            dest = kQInteract;
          }
        }
      } else {
        slot_load(S, e, ph, cw, idx);
        ph.can_enter = (int)((e.z >> kSlExcl) & 1u);
        sec.has = (int)((e.z >> kSlSec) & 1u);
        dest = kQFly;
        aim = event == kQFly && ph.t_exit < R<real>(0);
      }
      sec.tid = (int)(slot0 + (uint32_t)k);
      uint64_t key = args.seed, hid = args.h_begin + e.y;
      if constexpr (MULTI) {
        key = sg.sims[e.w].seed;
        hid = hid - sg.sims[e.w].h_begin;
      }
      const uint32_t h0 = (uint32_t)hid, h1 = (uint32_t)(hid >> 32), k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
      if (event == kQInteract) {
        pmat = (int)(cw >> 16);
        pscored = (int)((e.z >> kSlImage) & 1u);
        pv = real_bits(ph.t_exit);
        EventRng g{buf, ahead[threadIdx.x], k0, k1, 0u, h0, h1, e.x, idx};
        g.begin();
        real ed;
        int kind;
        const bool done = pool_interact(s, ph, g, &bc, sec, pmat, (e.z >> kSlRetry) != 0u, trials, kind, ed);
        g.end();
        e.x = g.blk;
        idx = g.idx;
        if (!done) {
          dest = kQInteract;
        } else if (pscored) {
          uint32_t v = pv;
          bool in = true;
          if constexpr (DG > 0) in = dose_voxel(s, ph.pos, v);
          if (in) {
            list_deposit(S.x, n_list, t, v, ed, n_dep, n_ent, n_over);
            if constexpr (DG == 2) {
              real dd = ed * s.drho_min;
              dd = dd / s.mat_rho[pmat];
              ld.deposit(td, v, dd);
            }
          }
          aim = ph.alive;
          if (!ph.alive) dest = kQRefill;
        } else {
          dest = ph.alive ? kQWorld : kQRefill;
          ph.can_enter = 1;
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
            const int r = dose_world_flight(s, ph, g, pmat, pscored);
            if (r == kRefill) ++n_esc;
            ph.t_exit = R<real>(-1);
            dest = r == kInteract ? kQInteract : (r == kFly ? kQFly : kQRefill);
          } else {
            ph.in_image = 1;
            const int r = image_flight(s, ph, g, pmat, pv, pscored, n_wood, n_real);
            dest = r == kInteract ? kQInteract : (ph.in_image ? kQFly : kQWorld);
          }
          g.end(buf, e.x, idx);
        }
      }
      if (dest == kQRefill && sec.has) {
        take_secondary(s, ph, sec);
        ph.t_exit = R<real>(-1);
        dest = ph.in_image ? kQFly : kQWorld;
        fresh = true;
      }
      // ---- the photon back into its slot
      const bool pend = dest == kQInteract;
      if (live) {
        slot_store(S, ph, pend, fresh, pmat, pv, trials);
        e.z = (uint32_t)ph.steps | ((uint32_t)idx << kSlIdx) | ((uint32_t)ph.can_enter << kSlExcl) |
              ((uint32_t)sec.has << kSlSec) | ((uint32_t)n_list << kSlList);
        if (pend) e.z |= (pscored ? 1u << kSlImage : 0u) | (trials ? 1u << kSlRetry : 0u);
      }
      if constexpr (DG == 2) e.w = (uint32_t)ld.n;
      S.e = e;
    }
    if (event == kQRefill) claims.advance(n);
    Q.put(dest, k, lane, lt_mask);
  }
  // ---- counters -------------------------------------------------------------
  unsigned long long *cnt = args.counters;
  warp_count(cnt + GG_CNT_WOODCOCK_STEPS, n_wood);
  warp_count(cnt + GG_CNT_REAL_INTERACTIONS, n_real);
  warp_count(cnt + GG_CNT_DEPOSITS, n_dep);
  warp_count(cnt + GG_CNT_WORLD_STEPS, n_world);
  warp_count(cnt + GG_CNT_TALLY_ENTRIES, n_ent);
  warp_count(cnt + GG_CNT_LIST_OVERFLOWS, n_over);
  warp_count(cnt + GG_CNT_ESCAPED, n_esc);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bc.loop_capped) atomicAdd(&cnt[GG_CNT_LOOP_CAPPED], (unsigned long long)bc.loop_capped);
    if (bc.stack_overflow) atomicAdd(&cnt[GG_CNT_STACK_OVERFLOW], (unsigned long long)bc.stack_overflow);
    if (bc.secondaries) atomicAdd(&cnt[GG_CNT_SECONDARIES], (unsigned long long)bc.secondaries);
  }
}

// Transport stage with the track-length estimator (a history scores every voxel
// it crosses: its list fills and empties many times, so it stays with its
// thread).  Persistent grid; each lane carries one history at a time
// and is in one of the states kRefill (needs a history), kFly (next event is
// a flight) or kInteract (a collision is pending).  Every iteration the block
// picks ONE phase from counts of its lanes' states - refill when at least
// refill_min lanes per warp wait for a history, interact when at least
// interact_min collisions per warp are pending, otherwise fly - and only the
// lanes in that state execute it.  Expensive code (source-record loads, tally
// flushes, Compton sampling) therefore runs with many lanes active instead of
// one lane at a time, all warps of a block execute the same code region at
// the same time (the kernel is bound by instruction fetch, not arithmetic),
// and the order of operations inside each history, hence its result, is
// unchanged.
// MINB = resident blocks per SM the register budget is sized for.
template <typename real, int MINB>
__global__ void __launch_bounds__(256, MINB) k_transport_tle(Scene<real> sg, KernelArgs args) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  __shared__ real sec_store[6 * 256];
  // ---- stage tables in shared memory --------------------------------------
  Scene<real> s = sg;
  {
    real *sh = reinterpret_cast<real *>(smem_raw);
    const int nsig = sg.n_comp * sg.n_e;
    real *ssig = sh;
    real *smaj = ssig + nsig;
    real *srho = smaj + sg.n_e;
    int *scomp = reinterpret_cast<int *>(srho + sg.n_mat);
    for (int i = threadIdx.x; i < nsig; i += blockDim.x) ssig[i] = sg.sig[i];
    for (int i = threadIdx.x; i < sg.n_e; i += blockDim.x) smaj[i] = sg.maj[i];
    for (int i = threadIdx.x; i < sg.n_mat; i += blockDim.x) {
      srho[i] = sg.mat_rho[i];
      scomp[i] = sg.mat_comp[i];
    }
    if (threadIdx.x == 0) bc = BlockCounters{0, 0, 0, 0, 0, 0, 0, 0};
    __syncthreads();
    s.sig = ssig;
    s.maj = smaj;
    s.mat_rho = srho;
    s.mat_comp = scomp;
  }
  const Records<real> rec = Records<real>::carve(args.records, args.rec_cap);
  Tally<real> t{args.acc_e, args.acc_e2};
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  const uint64_t n_hist = args.h_end - args.h_begin;
  __shared__ uint64_t wpool[kBlock / 32][2];  // per warp: claimed histories not yet handed out
  uint64_t *pool = wpool[threadIdx.x >> 5];
  if (lane == 0) pool[0] = pool[1] = 0;
  __syncwarp();

  Photon<real> ph;
  ph.alive = 0;
  Secondary<real> sec;
  sec.base = sec_store;
  sec.stride = blockDim.x;
  sec.tid = threadIdx.x;
  sec.has = 0;
  // history lists after the tables: [list][vox | acc][kHistList][blockDim.x]
  HistList<real> l;
  {
    const int nt = (int)blockDim.x;
    unsigned char *lists = smem_raw + transport_smem_bytes<real>(sg.n_comp, sg.n_e, sg.n_mat);
    l.vox = reinterpret_cast<uint32_t *>(lists) + threadIdx.x;
    l.acc = reinterpret_cast<real *>(lists + (size_t)kHistList * nt * sizeof(uint32_t)) + threadIdx.x;
    l.stride = nt;
    l.n = 0;
  }
  Event<real> ev;
  ev.clear();
  Rng g;
  int state = kRefill;
  bool in_hist = false;
  int pmat = 0, pscored = 0;
  uint32_t pv = 0;
  unsigned int n_wood = 0, n_real = 0, n_dep = 0, n_world = 0;

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
      // per-lane atomics: a warp-aggregated flush (same-voxel entries of the warp summed
      // first, __match_any_sync + shuffles) issued as many atomic instructions here and
      // made the transport 28 % slower, so it is not used
      if (need && in_hist) hlist_flush(l, t, &bc);
      if (need) in_hist = false;
      const uint64_t h = warp_pool_claim(pool, m_ref, lane, lt_mask, args.next, args.chunk);
      if (need) {
        if (h >= n_hist) {
          state = kDone;
        } else {
          const uint32_t f = rec.flags[h];
          const uint32_t rs = f & 3u;
          if (rs != kRecDead) {
            const uint64_t hid = args.h_begin + h;
            const uint64_t key = args.seed;
            ph.pos[0] = rec.px[h];
            ph.pos[1] = rec.py[h];
            ph.pos[2] = rec.pz[h];
            ph.dir[0] = rec.dx[h];
            ph.dir[1] = rec.dy[h];
            ph.dir[2] = rec.dz[h];
            set_energy(s, ph, rec.e[h]);
            ph.steps = (int)((f >> 2) & 1u);
            ph.alive = 1;
            ph.can_enter = 1;
            ph.in_head = 0;
            ph.exclude = -1;
            ph.w = s.s_fd_w;  // 1, or the forced direction's cone weight
            const uint32_t rp = rec.rng_pos[h];
            const uint4 b = rec.rng_buf[h];
            g.k0 = (uint32_t)key;
            g.k1 = (uint32_t)(key >> 32);
            g.stream = 0u;
            g.h0 = (uint32_t)hid;
            g.h1 = (uint32_t)(hid >> 32);
            g.blk = rp >> 3;
            g.idx = (int)(rp & 7u);
            g.buf[0] = b.x;
            g.buf[1] = b.y;
            g.buf[2] = b.z;
            g.buf[3] = b.w;
            if (rs == kRecInImage) {
              ph.in_image = 1;
              ph.t_exit = exit_distance(ph.pos, ph.dir, s.bmin, s.bmax);
              state = kFly;
            } else if (rs == kRecWorld) {
              ph.in_image = 0;
              state = kFly;
            } else {
              ph.in_image = 0;
              pmat = s.world_mat;
              pscored = 0;
              state = kInteract;
            }
            in_hist = true;
          }
        }
      }
    } else if (phase == kInteract) {
      if (state == kInteract) {
        state = do_interaction<real, false, true>(s, ph, g, &bc, pmat, pv, pscored, l, t, sec, n_dep, ev);
        if (state == kRefill && sec.has) {
          pop_secondary(s, ph, sec);
          state = kFly;
        }
      }
    } else {
      if (state == kFly) {
        state = flight<real, true>(s, ph, g, &bc, pmat, pv, pscored, n_wood, n_real, n_world,
                                   TleScore<real>{&l, &t, &n_dep});
        if (state == kRefill && sec.has) {
          pop_secondary(s, ph, sec);
          state = kFly;
        }
      }
    }
  }
  // ---- counters -------------------------------------------------------------
  unsigned long long *cnt = args.counters;
  auto warp_add = [&](unsigned int v, int slot) {
    unsigned long long x = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0 && x) atomicAdd(&cnt[slot], x);
  };
  warp_add(n_wood, GG_CNT_WOODCOCK_STEPS);
  warp_add(n_real, GG_CNT_REAL_INTERACTIONS);
  warp_add(n_dep, GG_CNT_DEPOSITS);
  warp_add(n_world, GG_CNT_WORLD_STEPS);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&cnt[GG_CNT_TALLY_ENTRIES], (unsigned long long)bc.tally_entries);
    atomicAdd(&cnt[GG_CNT_LIST_OVERFLOWS], (unsigned long long)bc.list_overflows);
    atomicAdd(&cnt[GG_CNT_ESCAPED], (unsigned long long)bc.escaped);
    atomicAdd(&cnt[GG_CNT_LOOP_CAPPED], (unsigned long long)bc.loop_capped);
    atomicAdd(&cnt[GG_CNT_STACK_OVERFLOW], (unsigned long long)bc.stack_overflow);
    atomicAdd(&cnt[GG_CNT_SECONDARIES], (unsigned long long)bc.secondaries);
  }
}

// Adds the per-batch fixed-point sums into the float64 images and clears them.
// scale multiplies the sums (1 for edep; 1 / rho_min for the dose tally, whose
// entries are edep * rho_min / rho), scale2 = scale^2 their squares.
__global__ void k_flush(unsigned long long *acc_e, unsigned long long *acc_e2, double *edep, double *edep2,
                        size_t n, double scale, double scale2) {
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    unsigned long long a = acc_e[i];
    if (a) {
      double v = (double)a * 2.3283064365386963e-10;
      v = v * scale;
      edep[i] += v;
      acc_e[i] = 0ull;
    }
    if (acc_e2) {
      const ulonglong2 b = reinterpret_cast<const ulonglong2 *>(acc_e2)[i];  // (low 32 bits, rest)
      if (b.x | b.y) {
        double lo = (double)b.x;
        lo = lo * 5.421010862427522e-20;  // 2^-64
        double hi = (double)b.y;
        hi = hi * 2.3283064365386963e-10;  // 2^-32
        double v = hi + lo;
        v = v * scale2;
        edep2[i] += v;
        reinterpret_cast<ulonglong2 *>(acc_e2)[i] = make_ulonglong2(0ull, 0ull);
      }
    }
  }
}


template <typename real>
size_t record_bytes(size_t cap) {
  return cap * (sizeof(uint4) + 7 * sizeof(real) + 3 * sizeof(uint32_t));
}

template <typename real>
cudaError_t launch_generate(const Scene<real> &s, const KernelArgs &a, cudaStream_t st) {
  uint64_t n = a.h_end - a.h_begin;
  unsigned int blocks = (unsigned int)((n + 255) / 256);
  if (s.n_sims > 0) k_generate<real, true><<<blocks, 256, 0, st>>>(s, a);
  else k_generate<real, false><<<blocks, 256, 0, st>>>(s, a);
  return cudaGetLastError();
}

template <typename real, bool MULTI, int DG>
static cudaError_t launch_pool_v(const Scene<real> &s, const KernelArgs &a, const PoolPlan &p, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_transport_pool<real, MULTI, DG>, 227 * 1024, configured);
  if (e != cudaSuccess) return e;
  k_transport_pool<real, MULTI, DG><<<p.grid, p.block, p.smem, st>>>(s, a, p.slots);
  return cudaGetLastError();
}

template <typename real, int MINB>
static cudaError_t launch_tle_v(const Scene<real> &s, const KernelArgs &a, int grid, int block, size_t smem,
                                cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_transport_tle<real, MINB>, kTransportSmemMax, configured);
  if (e != cudaSuccess) return e;
  smem += hist_list_bytes<real>(1, block);
  if (smem > (size_t)kTransportSmemMax) return cudaErrorInvalidValue;
  k_transport_tle<real, MINB><<<grid, block, smem, st>>>(s, a);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_transport(const Scene<real> &s, const KernelArgs &a, const PoolPlan &p, cudaStream_t st) {
  // SPECT runs use the stage kernels of gg_spect.cu, the track-length estimator launch_transport_tle
  if (s.spect || s.muen || p.block <= 0 || p.block > PoolShape<real>::kBlock || p.slots < 8 || p.slots > PoolShape<real>::kRing) return cudaErrorInvalidValue;
  if (s.dgrid) {
    // dose grid of its own (single simulations, analog scoring)
    if (s.n_sims > 0) return cudaErrorInvalidValue;
    return s.ddose ? launch_pool_v<real, false, 2>(s, a, p, st) : launch_pool_v<real, false, 1>(s, a, p, st);
  }
  return s.n_sims > 0 ? launch_pool_v<real, true, 0>(s, a, p, st) : launch_pool_v<real, false, 0>(s, a, p, st);
}

template <typename real>
cudaError_t launch_transport_tle(const Scene<real> &s, const KernelArgs &a, int grid, int block, size_t smem, int minb,
                                 cudaStream_t st) {
  // single simulations on the image grid only
  if (s.spect || !s.muen || s.dgrid || s.n_sims > 0 || block <= 0 || block > kBlock) return cudaErrorInvalidValue;
  if (minb <= 2) return launch_tle_v<real, 2>(s, a, grid, block, smem, st);
  if (minb == 3) return launch_tle_v<real, 3>(s, a, grid, block, smem, st);
  return launch_tle_v<real, 4>(s, a, grid, block, smem, st);
}

cudaError_t launch_flush(unsigned long long *acc_e, unsigned long long *acc_e2, double *edep, double *edep2,
                         size_t n, int grid, cudaStream_t st, double scale) {
  k_flush<<<grid, 256, 0, st>>>(acc_e, acc_e2, edep, edep2, n, scale, scale * scale);
  return cudaGetLastError();
}

template <typename real>
cudaError_t tle_occupancy(int block, size_t smem, int minb, int *bps) {
  smem += hist_list_bytes<real>(1, block);
  if (minb <= 2) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_transport_tle<real, 2>, block, smem);
  if (minb == 3) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_transport_tle<real, 3>, block, smem);
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bps, k_transport_tle<real, 4>, block, smem);
}

// Launch shape of a pooled run: one block per SM.  More slots per thread keep
// the rounds full, so they take all shared memory beside the tables, but no
// more than the run has histories for.  block, blocks: most threads per block
// and resident blocks per SM (of 256 threads) of the options, 0 for the
// kernel's register budget; slot_bytes, scratch_bytes: of one slot, shared and global.
template <typename real>
cudaError_t pool_plan(int device, size_t table_bytes, int block, int blocks, uint64_t n_hist, size_t slot_bytes,
                      size_t scratch_bytes, PoolPlan *p) {
  int n_sm = 0, optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e != cudaSuccess) return e;
  using Shape = PoolShape<real>;
  constexpr int kGang = 32 * Shape::kGang;
  const uint64_t per_sm = (n_hist + n_sm - 1) / n_sm;
  int threads = Shape::kBlock;
  if (blocks > 0) threads = std::min(threads, 256 * blocks);
  if (block > 0) threads = std::min(threads, block);
  threads = (int)std::min<uint64_t>(threads, (per_sm + 31) / 32 * 32);
  const size_t slot = slot_bytes, fixed = pool_static<real>() + table_bytes;
  const int room = (size_t)optin > fixed ? (int)(((size_t)optin - fixed) / slot) : 0;
  while (threads > kGang && room < threads) threads -= kGang;  // (large tables: fewer gangs)
  const int gangs = (threads + kGang - 1) / kGang;
  const int most = std::min(room / gangs, Shape::kRing - 32) / 8 * 8;
  if (most < 8) return cudaErrorInvalidValue;
  const uint64_t share = std::max<uint64_t>((per_sm + gangs - 1) / gangs, 32);
  p->grid = n_sm;
  p->block = threads;
  p->gangs = gangs;
  p->slots = (int)std::min<uint64_t>(most, (share + 7) / 8 * 8);
  p->smem = slot * p->slots * gangs + table_bytes;
  p->scratch = (size_t)p->grid * gangs * p->slots * scratch_bytes;
  return cudaSuccess;
}

template <typename real>
size_t dose_slot_bytes() {
  return sizeof(DoseSlot<real>);
}
template <typename real>
size_t slot_scratch_bytes(bool two) {
  return 6 * sizeof(real) + (two ? kHistList * (sizeof(real) + sizeof(uint32_t)) : 0);
}

// Histories a gang claims at a time: an even share of a small run, else the
// per-warp chunk of the options for each of its warps.
int pool_chunk(const PoolPlan &p, int chunk, uint64_t n_hist) {
  const uint64_t gangs = (uint64_t)p.grid * p.gangs, share = (n_hist + gangs - 1) / gangs;
  const uint64_t warps = (uint64_t)std::max(p.block / 32 / p.gangs, 1);
  return (int)std::max<uint64_t>(32, std::min<uint64_t>(share, warps * std::min(chunk, 1 << 20)));
}

template size_t record_bytes<float>(size_t);
template size_t record_bytes<double>(size_t);
template cudaError_t launch_generate<float>(const Scene<float> &, const KernelArgs &, cudaStream_t);
template cudaError_t launch_generate<double>(const Scene<double> &, const KernelArgs &, cudaStream_t);
template cudaError_t launch_transport<float>(const Scene<float> &, const KernelArgs &, const PoolPlan &, cudaStream_t);
template cudaError_t launch_transport<double>(const Scene<double> &, const KernelArgs &, const PoolPlan &,
                                              cudaStream_t);
template cudaError_t launch_transport_tle<float>(const Scene<float> &, const KernelArgs &, int, int, size_t, int,
                                                 cudaStream_t);
template cudaError_t launch_transport_tle<double>(const Scene<double> &, const KernelArgs &, int, int, size_t, int,
                                                  cudaStream_t);
template cudaError_t pool_plan<float>(int, size_t, int, int, uint64_t, size_t, size_t, PoolPlan *);
template cudaError_t pool_plan<double>(int, size_t, int, int, uint64_t, size_t, size_t, PoolPlan *);
template size_t dose_slot_bytes<float>();
template size_t dose_slot_bytes<double>();
template size_t slot_scratch_bytes<float>(bool);
template size_t slot_scratch_bytes<double>(bool);
template cudaError_t tle_occupancy<float>(int, size_t, int, int *);
template cudaError_t tle_occupancy<double>(int, size_t, int, int *);

}  // namespace gg
