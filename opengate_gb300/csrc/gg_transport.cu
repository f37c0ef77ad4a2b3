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
//     runs one kind of event at a time on full warps (gg_pool.cuh);
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
#include <type_traits>

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
    __shared__ uint8_t waiting[256 / 32][32];
    int st = warp_iso_direction_accepted(s, g, ph, live, &bc, waiting[threadIdx.x >> 5]);
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
// histories to 6 MeV, 47.1 -> 29.9 ms against one photon per thread with block-wide phases
// (204 warp instructions per history at 21 active lanes; 379 at 8.6); 24
// batched simulations 21.0 -> 12.2 ms, FP64 8.9 -> 4.1 ms per 1e6.
// MULTI: batched simulations; DG: dose tally on a grid of its own (1: edep,
// 2: edep and dose), Scene::dgrid; TLE: track-length estimator
// (GateTLEDoseActor::ScoreTLEDepositStep,
// core/opengate_core/opengate_lib/GateTLEDoseActor.cpp:249-299): a photon at or
// below its threshold energy scores e * mu_en(E, material) * length in every
// voxel its flights cross, and its interactions deposit nothing
// (GateTLEDoseActor.cpp:236-243).  Such a flight is two kinds of event: its path
// is drawn, then walked kTleSteps boundaries a round.  64^3 voxels of 2 mm,
// 3e6 photons of 1 MeV in a pencil beam (81 voxels each): 13.5 -> 6.5 ms
// against one photon per thread with each path walked at once (2088 warp
// instructions per history at 7.4 lanes; now 880 at 25).  Two things count
// together: without the sums of equal voxels (lists_flush_same) the atomics of
// the beam's axis queue at a few L2 slices, 12.2 ms.
template <typename real, bool MULTI, int DG, bool TLE>
__global__ void __launch_bounds__(PoolShape<real>::kBlock, 1) k_transport_pool(Scene<real> sg, KernelArgs args, int n_slots, int gang_threads) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BlockCounters bc;
  using Shape = PoolShape<real>;
  using Slot = std::conditional_t<TLE, TleSlot<real>, std::conditional_t<DG == 2, GridSlot<real>, DoseSlot<real>>>;
  constexpr int kGangs = Shape::kGangs;
  constexpr int kNq = TLE ? kTleQueues : kQueues;
  using Queues = EventQueues<Shape::kRing, kNq>;
  __shared__ __align__(16) unsigned push[kGangs][3 * Queues::kSet];
  __shared__ __align__(16) uint32_t ahead[Shape::kBlock][4];  // EventRng's second block of each thread
  __shared__ uint16_t ring[kGangs][kNq * Shape::kRing];
  __shared__ unsigned long long s_claim[kGangs];
  Scene<real> s = sg;
  const unsigned lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  const int gang = (int)threadIdx.x / gang_threads, gang0 = gang * gang_threads;
  const int gangs = ((int)blockDim.x + gang_threads - 1) / gang_threads;
  // dynamic shared memory: slots of the gangs, tables
  Slot *const slots = reinterpret_cast<Slot *>(smem_raw) + gang * n_slots;
  Queues Q;
  Q.init(gang, threadIdx.x - (unsigned)gang0, min((unsigned)gang_threads, blockDim.x - (unsigned)gang0), ring[gang], push[gang],
         (unsigned)n_slots);
  for (int i = (int)Q.tid; i < n_slots; i += (int)Q.size) slots[i].e = make_uint4(0u, 0u, 0u, 0u);
  stage_tables(sg, s, smem_raw + sizeof(Slot) * (size_t)(gangs * n_slots), bc);

  const Records<real> rec = Records<real>::carve(args.records, args.rec_cap);
  Tally<real> t{args.acc_e, args.acc_e2};
  const Tally<real> td{args.acc_d, args.acc_d2};
  const uint32_t n_hist = (uint32_t)(args.h_end - args.h_begin);
  const uint32_t slot0 = (blockIdx.x * (uint32_t)gangs + (uint32_t)gang) * (uint32_t)n_slots;
  const uint32_t all_slots = gridDim.x * (uint32_t)(gangs * n_slots);  // global scratch: one column per slot
  Secondary<real> sec;
  sec.base = reinterpret_cast<real *>(args.slot_scratch);
  sec.stride = (int)all_slots;
  // an entry of a slot's list into the tallies
  auto list_entry = [&](const Slot &S, int k) {
    if constexpr (MULTI) tally_entry(tally_at(args, sg.sims[S.e.w].vox_off, real(0)), S.x.vox[k], S.x.acc[k]);
    else tally_entry(t, S.x.vox[k], S.x.acc[k]);
    if constexpr (DG == 2) tally_entry(td, S.x.vox[k], S.x.dose[k]);
  };
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
      const int n_old = k >= 0 ? (int)((slots[k].e.z >> kSlList) & 15u) : 0;
      if constexpr (TLE) {
        lists_flush_same(slots[max(k, 0)].x, n_old, t, lane);
        n_ent += (unsigned)n_old;
      } else {
        lists_flush(slots, max(k, 0), n_old, reinterpret_cast<uint16_t *>(ahead[threadIdx.x & ~31u]), lane,
                    list_entry, n_ent);
      }
    }
    if constexpr (TLE) {
      if (event == kQWalk) {
        dest = tle_walk(s, slots, k, lane, t, n_dep, n_ent, n_over);
        Q.put(dest, k, lane, lt_mask);
        continue;
      }
    }
    if (k >= 0) {
      Slot &S = slots[k];
      uint4 e = S.e;
      int n_list = (int)((e.z >> kSlList) & 15u);
      auto bind = [&](uint32_t sim) {  // batched simulations: the history's geometry, majorant and tally
        const SimDesc<real> &d = sg.sims[sim];
        bind_geometry(s, d, sg.labels, sg.sim_maj + (size_t)sim * sg.n_e);
        t = tally_at(args, d.vox_off, real(0));
      };
      if constexpr (MULTI) bind(e.w);
      auto here = [&](int q) {  // (t is the bound simulation's)
        tally_entry(t, S.x.vox[q], S.x.acc[q]);
        if constexpr (DG == 2) tally_entry(td, S.x.vox[q], S.x.dose[q]);
      };
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
          // in the image, or at the collision in the world that ended the source stage's flight
          // (without a branch: 24 batched simulations 12.5 -> 12.2 ms, CT 30.4 -> 30.1)
          aim = (f & 3u) == kRecInImage;
          dest = aim ? kQFly : kQInteract;
          pmat = s.world_mat;
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
        const bool score = !TLE || ph.e > s.tle_thr;
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
          if constexpr (TLE) in = score;
          if (in) {
            const int n_before = n_list;
            const int at = list_deposit(S.x, n_list, v, ed, n_dep, n_ent, n_over, here);
            if constexpr (DG == 2) {
              if (at >= 0) {
                real dd = ed * s.drho_min;
                dd = dd / s.mat_rho[pmat];
                S.x.dose[at] = n_list == n_before ? S.x.dose[at] + dd : dd;  // (one entry more, or only it after a flush)
              }
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
        TwoWords g;
        g.draw(buf, e.x, idx, 0u, h0, h1, k0, k1);
        if constexpr (TLE) {
          if (event == kQFly && e.w) {  // a scored path has been walked; no collision: the next flight
            e.w = 0u;
            ph.in_image = 1;
            const int r = image_arrive(s, ph, g, S.x.td.w, pmat, pv, pscored, n_wood, n_real);
            dest = r == kInteract ? kQInteract : (ph.in_image ? kQFly : kQWorld);
          }
        }
        if (TLE && event != kQWorld && dest != kQFly) {
          g.end(buf, e.x, idx);
        } else if (++ph.steps > kStepCap) {
          atomicAdd(&bc.loop_capped, 1u);
          if constexpr (TLE) g.end(buf, e.x, idx);
          dest = kQRefill;
        } else {
          if (event == kQWorld) {
            ++n_world;
            const int r = dose_world_flight(s, ph, g, pmat, pscored);
            if (r == kRefill) ++n_esc;
            ph.t_exit = R<real>(-1);
            dest = r == kInteract ? kQInteract : (r == kFly ? kQFly : kQRefill);
          } else if (TLE && ph.e <= s.tle_thr) {
            if (ph.e <= s.tle_emin) {  // the kill energy: the rest is left where the photon is
              list_deposit(S.x, n_list, voxel_of(s, ph.pos), ph.e, n_dep, n_ent, n_over, here);
              dest = kQRefill;
            } else {
              if constexpr (TLE) {
                VoxelWalk<real> w;
                w.start(s, ph.pos, ph.dir);
                tle_store(S.x, w, woodcock_path(ph, g));
              }
              e.w = 1u;
              dest = kQWalk;
            }
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

template <typename real, bool MULTI, int DG, bool TLE = false>
static cudaError_t launch_pool_v(const Scene<real> &s, const KernelArgs &a, const PoolPlan &p, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_transport_pool<real, MULTI, DG, TLE>, 227 * 1024, configured);
  if (e != cudaSuccess) return e;
  k_transport_pool<real, MULTI, DG, TLE><<<p.grid, p.block, p.smem, st>>>(s, a, p.slots, p.gang_threads);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_transport(const Scene<real> &s, const KernelArgs &a, const PoolPlan &p, cudaStream_t st) {
  // SPECT runs use the stage kernels of gg_spect.cu
  if (s.spect || p.block <= 0 || p.block > PoolShape<real>::kBlock || p.slots < 8 || p.slots > PoolShape<real>::kRing) return cudaErrorInvalidValue;
  if (s.muen) {  // track-length estimator: single simulations on the image grid only
    if (s.dgrid || s.n_sims > 0) return cudaErrorInvalidValue;
    return launch_pool_v<real, false, 0, true>(s, a, p, st);
  }
  if (s.dgrid) {
    // dose grid of its own (single simulations, analog scoring)
    if (s.n_sims > 0) return cudaErrorInvalidValue;
    return s.ddose ? launch_pool_v<real, false, 2>(s, a, p, st) : launch_pool_v<real, false, 1>(s, a, p, st);
  }
  return s.n_sims > 0 ? launch_pool_v<real, true, 0>(s, a, p, st) : launch_pool_v<real, false, 0>(s, a, p, st);
}

cudaError_t launch_flush(unsigned long long *acc_e, unsigned long long *acc_e2, double *edep, double *edep2,
                         size_t n, int grid, cudaStream_t st, double scale) {
  k_flush<<<grid, 256, 0, st>>>(acc_e, acc_e2, edep, edep2, n, scale, scale * scale);
  return cudaGetLastError();
}

template <typename real>
cudaError_t pool_plan(int device, size_t table_bytes, int blocks, uint64_t n_hist, size_t slot_bytes,
                      size_t scratch_bytes, int queues, PoolPlan *p) {
  int n_sm = 0, optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e != cudaSuccess) return e;
  return pool_shape<real>(n_sm, (size_t)optin, table_bytes, blocks, n_hist, slot_bytes, scratch_bytes, queues, p)
             ? cudaSuccess
             : cudaErrorInvalidValue;
}

template <typename real>
size_t dose_slot_bytes(bool tle, bool two) {
  return tle ? sizeof(TleSlot<real>) : (two ? sizeof(GridSlot<real>) : sizeof(DoseSlot<real>));
}
template <typename real>
size_t slot_scratch_bytes() {
  return 6 * sizeof(real);
}

template size_t record_bytes<float>(size_t);
template size_t record_bytes<double>(size_t);
template cudaError_t launch_generate<float>(const Scene<float> &, const KernelArgs &, cudaStream_t);
template cudaError_t launch_generate<double>(const Scene<double> &, const KernelArgs &, cudaStream_t);
template cudaError_t launch_transport<float>(const Scene<float> &, const KernelArgs &, const PoolPlan &, cudaStream_t);
template cudaError_t launch_transport<double>(const Scene<double> &, const KernelArgs &, const PoolPlan &,
                                              cudaStream_t);
template cudaError_t pool_plan<float>(int, size_t, int, uint64_t, size_t, size_t, int, PoolPlan *);
template cudaError_t pool_plan<double>(int, size_t, int, uint64_t, size_t, size_t, int, PoolPlan *);
template size_t dose_slot_bytes<float>(bool, bool);
template size_t dose_slot_bytes<double>(bool, bool);
template size_t slot_scratch_bytes<float>();
template size_t slot_scratch_bytes<double>();

}  // namespace gg
