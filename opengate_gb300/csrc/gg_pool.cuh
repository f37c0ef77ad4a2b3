// gg_pool.cuh - photon slots and event queues of the pooled transport kernels.
//
// A gang of warps owns more photon slots than it has threads; their whole
// state lives in shared memory, with one queue of slot numbers per kind of next
// event.  Every round the gang picks its longest queue, each thread takes one
// slot of it, runs that event, stores the photon back and appends the slot to
// the queue of the photon's next event.  Nearly every lane of a round has a
// photon: one photon per thread instead kept 8.6 of 32 lanes active, since a
// lane could only wait for its own photon's kind of event to come up.
//
// The warps of a gang run one code region at a time because the kernels are
// sensitive to instruction fetch; the gangs of a block share its tables and
// run on their own, so one gang's barrier is covered by the others.
//
// One barrier per round: the pushes of round k are counted in push[(k + 1) % 3]
// and read by every thread after the barrier that opens round k + 1; the set
// of the round after is cleared meanwhile.  A round takes no more entries than
// its ring has free, so its pushes never overwrite an entry that a slower warp
// still has to read.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_device.cuh"
#include "gg_internal.h"
#include "gg_physics.cuh"
#include "gg_tc.cuh"

namespace gg {

// kQWalk: the track-length estimator's only
enum : int { kQRefill = 0, kQFly = 1, kQWorld = 2, kQInteract = 3, kQueues = 4, kQWalk = 4, kTleQueues = 5, kQNone = 8 };
// A gang's event queues.  cnt / tail are the same in every thread: queue
// lengths and ring positions, 16 bits each (queue q in half q & 1 of word q >> 1).
template <int kPoolRing, int NQ = kQueues>
struct EventQueues {
  static constexpr int kWords = (NQ + 1) / 2, kSet = NQ <= 4 ? 4 : 8;  // kSet: words of a push set
  static_assert(NQ <= 6, "round() and put() select among three words");
  static_assert((kPoolRing & (kPoolRing - 1)) == 0 && kPoolRing <= 1024, "ring positions are masked, packed in 16 bits");
  uint16_t *ring;     // [NQ][kPoolRing]
  unsigned *push;     // [3][kSet]
  unsigned cnt[kWords], tail[kWords];
  unsigned rd;        // push set of this round's barrier, rotates through 0, 1, 2
  unsigned tid, size; // the thread in its gang, the gang's threads
  int bar;            // named barrier

  // every slot waits for a history; the caller's next round() opens with the barrier
  __device__ __forceinline__ void init(int gang, unsigned t, unsigned n, uint16_t *r, unsigned *p, unsigned slots) {
    tid = t;
    size = n;
    bar = 1 + gang;
    ring = r;
    push = p;
    for (unsigned i = tid; i < slots; i += size) ring[kQRefill * kPoolRing + i] = (uint16_t)i;
    if (tid < 3 * kSet) push[tid] = 0u;
#pragma unroll
    for (int w = 0; w < kWords; ++w) cnt[w] = tail[w] = 0u;
    cnt[0] = slots;  // (kQRefill is queue 0)
    tail[0] = slots & (kPoolRing - 1u);
    rd = 0u;
  }
  __device__ __forceinline__ void sync() const { named_bar(bar, (int)size); }

  // The event of this round (kQNone: no slot is left) and the thread's slot
  // (-1: none); n: threads that have one.
  __device__ __forceinline__ int round(int &slot, unsigned &n) {
    constexpr unsigned kMask = (kPoolRing - 1u) * 0x10001u;
    sync();
    const unsigned clr = rd == 0u ? 2u : rd - 1u;  // (rd + 2) % 3: the set after next
    unsigned best = 0u;                            // the longest queue: length * 8 + queue
#pragma unroll
    for (int h = 0; h < kSet / 4; ++h) {
      const uint4 p = reinterpret_cast<const uint4 *>(push + rd * kSet)[h];
      if (tid == 0) reinterpret_cast<uint4 *>(push + clr * kSet)[h] = make_uint4(0u, 0u, 0u, 0u);
      const unsigned add[2] = {p.x | (p.y << 16), p.z | (p.w << 16)};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int w = 2 * h + j;
        if (w < kWords) {
          cnt[w] += add[j];
          tail[w] = (tail[w] + add[j]) & kMask;
          best = max(best, max(((cnt[w] & 0xffffu) << 3) | (2u * w), ((cnt[w] >> 13) & ~7u) | (2u * w + 1u)));
        }
      }
    }
    rd = rd == 2u ? 0u : rd + 1u;  // the set this round pushes to
    const unsigned q = best & 7u, len = best >> 3, sh = (q & 1u) << 4;
    n = min(min(len, size), (unsigned)kPoolRing - len);
    slot = -1;
    if (len == 0u) return kQNone;
    const unsigned head = (tail_word((int)q) >> sh) - len;
    if (tid < n) slot = ring[q * kPoolRing + ((head + tid) & (kPoolRing - 1u))];
#pragma unroll
    for (int w = 0; w < kWords; ++w)
      if ((int)(q >> 1) == w) cnt[w] -= n << sh;
    return (int)q;
  }

  __device__ __forceinline__ unsigned tail_word(int q) const {
    if (NQ > 4 && (q & 4)) return tail[kWords - 1];
    return q & 2 ? tail[1] : tail[0];
  }

  // Appends the lane's slot to queue `dest` (kQNone: nowhere); every lane of the warp calls it.
  __device__ __forceinline__ void put(int dest, int slot, unsigned lane, unsigned lt_mask) {
    const unsigned b0 = __ballot_sync(0xffffffffu, dest == 0), b1 = __ballot_sync(0xffffffffu, dest == 1),
                   b2 = __ballot_sync(0xffffffffu, dest == 2), b3 = __ballot_sync(0xffffffffu, dest == 3);
    unsigned m = dest & 2 ? (dest & 1 ? b3 : b2) : (dest & 1 ? b1 : b0);
    if constexpr (NQ > 4) {
      const unsigned b4 = __ballot_sync(0xffffffffu, dest == 4);
      if (dest == 4) m = b4;
    }
    const unsigned rank = __popc(m & lt_mask);
    unsigned off = 0u;
    if (dest < NQ && rank == 0u) off = atomicAdd(&push[rd * kSet + (unsigned)dest], __popc(m));
    off = __shfl_sync(0xffffffffu, off, __ffs(m) - 1);  // (the lane's own value is unused when m is 0)
    const unsigned t = tail_word(dest) >> ((dest & 1) << 4);
    if (dest < NQ) ring[(unsigned)dest * kPoolRing + ((t + off + rank) & (kPoolRing - 1u))] = (uint16_t)slot;
  }
};

// Four reals that move as 16-byte words.
template <typename real>
struct alignas(16) Real4 {
  real x, y, z, w;
};
__device__ __forceinline__ float bits_real(float, uint32_t u) { return __uint_as_float(u); }
__device__ __forceinline__ double bits_real(double, uint32_t u) { return __longlong_as_double((long long)u); }
__device__ __forceinline__ uint32_t real_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t real_bits(double v) { return (uint32_t)__double_as_longlong(v); }

// meta word of a slot: steps (20 bits) | words of the Philox buffer used (3) |
// exclude + 1 (2) | pending interaction in the image (1) | waiting secondary
// (1) | list length (4) | Compton sampling not finished (1)
constexpr uint32_t kSlSteps = (1u << 20) - 1u;
constexpr int kSlIdx = 20, kSlExcl = 23, kSlImage = 25, kSlSec = 26, kSlList = 27, kSlRetry = 31;
static_assert(kStepCap < (1 << 20), "the step count has 20 bits in the slot's meta word");
static_assert(kHistList < 16, "the list length has 4 bits in the slot's meta word");

// A photon slot in shared memory.  a: position, path to the image boundary
// (negative: not known; a pending interaction: its voxel); b: direction,
// energy; c: majorant (Compton sampling not finished: rejected trials), its
// inverse, energy-grid fraction, energy index | material << 16; rng: the Philox
// block being drawn from; e: next block, history (record), meta, a word of the
// kernel's own; X: more of its own.  The stride is an odd number of 16-byte
// words, so slots spread over the banks.
template <typename real, typename X>
struct PhotonSlot {
  Real4<real> a, b, c;
  uint4 rng, e;
  X x;
};

// A slot's photon into registers.
template <typename real, typename Slot>
__device__ __forceinline__ void slot_load(const Slot &S, const uint4 &e, Photon<real> &ph, uint32_t &cw, int &idx) {
  const Real4<real> a = S.a, b = S.b, c = S.c;
  cw = real_bits(c.w);
  ph.pos[0] = a.x;
  ph.pos[1] = a.y;
  ph.pos[2] = a.z;
  ph.dir[0] = b.x;
  ph.dir[1] = b.y;
  ph.dir[2] = b.z;
  ph.e = b.w;
  ph.t_exit = a.w;
  ph.mumax = c.x;
  ph.inv_mumax = c.y;
  ph.ei.fe = c.z;
  ph.ei.ie = (int)(cw & 0xffffu);
  ph.steps = (int)(e.z & kSlSteps);
  idx = (int)((e.z >> kSlIdx) & 7u);
}

// ... and back: pend: an interaction in pmat (voxel pv) is pending; fresh:
// direction and energy changed; trials: of a Compton sampling not finished.
template <typename real, typename Slot>
__device__ __forceinline__ void slot_store(Slot &S, const Photon<real> &ph, bool pend, bool fresh, int pmat,
                                           uint32_t pv, uint32_t trials) {
  S.a = Real4<real>{ph.pos[0], ph.pos[1], ph.pos[2], pend ? bits_real(real(0), pv) : ph.t_exit};
  const uint32_t cw = (uint32_t)ph.ei.ie | ((uint32_t)pmat << 16);
  if (fresh) {
    S.b = Real4<real>{ph.dir[0], ph.dir[1], ph.dir[2], ph.e};
    S.c = Real4<real>{trials ? bits_real(real(0), trials) : ph.mumax, ph.inv_mumax, ph.ei.fe,
                      bits_real(real(0), cw)};
  } else if (pend) {
    S.c.w = bits_real(real(0), cw);
  }
}

// Items (records, queue entries) claimed from the launch's work counter and not
// yet handed out; the same in every thread of a gang.
struct ItemClaims {
  uint32_t next, end, avail, base, got;
  bool exhausted;

  __device__ __forceinline__ void init() {
    next = end = 0u;
    exhausted = false;
  }
  // the next n items, one per thread in order (coalesced loads), claiming `chunk` more when short
  template <typename Queues>
  __device__ __forceinline__ void take(const Queues &q, unsigned n, unsigned long long *counter, int chunk,
                                       uint32_t n_items, unsigned long long *s_claim) {
    avail = end - next;
    base = got = 0u;
    if (avail < n && !exhausted) {
      if (q.tid == 0) *s_claim = atomicAdd(counter, (unsigned long long)chunk);
      q.sync();
      const unsigned long long c = *s_claim;
      if (c < n_items) {
        base = (uint32_t)c;
        got = min((uint32_t)chunk, n_items - base);
      }
      exhausted = c + (unsigned long long)chunk >= n_items;
    }
  }
  // thread r's item; false: none is left now
  __device__ __forceinline__ bool item(uint32_t r, uint32_t &h) const {
    h = r < avail ? next + r : base + (r - avail);
    return r < avail || r - avail < got;
  }
  __device__ __forceinline__ void advance(unsigned n) {
    if (n <= avail) {
      next += n;
    } else {
      next = base + min(n - avail, got);
      end = base + got;
    }
  }
};

// The stream of one event: the slot's block (words idx .. 3 left) and the one
// after it, made when the event begins while the warp is converged, so the
// draws inside divergent code seldom call the generator.  The words live in
// shared memory (a register window would be selected word by word); reserve(n)
// comes before n draws.
struct EventRng {
  uint32_t *buf, *nxt;  // the slot's block, the thread's own block
  uint32_t k0, k1, stream, h0, h1;
  uint32_t blk;         // number of nxt's block
  int idx;              // 0 .. 8: words used of buf, nxt

  __device__ __forceinline__ void begin() {
    *reinterpret_cast<uint4 *>(nxt) = philox_block(blk, stream, h0, h1, k0, k1);
  }
  // nxt becomes the slot's block
  __device__ __forceinline__ void shift() {
    *reinterpret_cast<uint4 *>(buf) = *reinterpret_cast<const uint4 *>(nxt);
    blk += 1u;
    idx -= 4;
  }
  __device__ __forceinline__ void reserve(int n) {
    if (idx + n > 8) {
      shift();
      begin();
    }
  }
  __device__ __forceinline__ uint32_t next() {
    const uint32_t v = idx < 4 ? buf[idx] : nxt[idx - 4];
    ++idx;
    return v;
  }
  // the slot's state after the event: nxt becomes its block when words of it are drawn
  __device__ __forceinline__ void end() {
    if (idx > 4) shift();
  }
};

// The one or two words of a flight, drawn while the warp is converged: at most
// one block is made, by the lanes whose buffer runs out.
struct TwoWords {
  uint32_t w[2];
  uint4 nb;
  int used;

  __device__ __forceinline__ void draw(const uint32_t *buf, uint32_t blk, int idx, uint32_t stream, uint32_t h0,
                                       uint32_t h1, uint32_t k0, uint32_t k1) {
    if (idx > 2) nb = philox_block(blk, stream, h0, h1, k0, k1);
    w[0] = idx < 4 ? buf[idx & 3] : nb.x;
    w[1] = idx < 3 ? buf[(idx + 1) & 3] : (idx == 3 ? nb.x : nb.y);
    used = 0;
  }
  __device__ __forceinline__ uint32_t next() {
    const uint32_t v = used == 0 ? w[0] : w[1];
    ++used;
    return v;
  }
  // the slot's state after `used` draws
  __device__ __forceinline__ void end(uint32_t *buf, uint32_t &blk, int &idx) const {
    idx += used;
    if (idx > 4) {
      *reinterpret_cast<uint4 *>(buf) = nb;
      blk += 1u;
      idx -= 4;
    }
  }
};

// Compton trials of one interaction event; a photon that is rejected as often
// waits for the next event with the photons it meets there, instead of keeping
// its warp in the loop (a third of the trials fail; the worst of 32 lanes takes
// five or six).
constexpr int kKnTrials = 2;

// The interaction of a photon in material pmat (interact(): select_kind, then
// the process).  False: its Compton sampling is not finished, `trials` rejected
// so far; retry: it is such a photon.  ed: energy deposited locally.
template <typename real>
__device__ __forceinline__ bool pool_interact(const Scene<real> &s, Photon<real> &ph, EventRng &g, BlockCounters *bc,
                                              Secondary<real> &sec, int pmat, bool retry, uint32_t &trials, int &kind,
                                              real &ed) {
  kind = retry ? kCompton : select_kind(s, ph, pmat, g);
  ed = R<real>(0);
  bool done = true;
  real cost = R<real>(1), st2 = R<real>(0), eps = R<real>(1);
  if (kind == kCompton) {
    const KleinNishina<real> kn(ph.e);
    trials = retry ? real_bits(ph.mumax) : 0u;
    real onecost;
    int left = kKnTrials;
#pragma unroll 1
    do {
      done = kn.trial(g, eps, onecost, st2);
      if (!done && ++trials >= (uint32_t)kLoopCap) {
        atomicAdd(&bc->loop_capped, 1u);
        done = true;
      }
    } while (!done && --left > 0);
    cost = R<real>(1) - onecost;
  } else if (kind == kPhoto) {
    ph.alive = 0;
    ed = ph.e;
  } else if (kind == kRayleigh) {
    cost = rayleigh_cost(s, s.mat_comp[pmat], ph, g, bc);
    st2 = rayleigh_sint2(cost);
  } else {
    ed = pair_conversion(s, ph, g, bc, sec);
  }
  if (done && (kind == kCompton || kind == kRayleigh)) scatter_dir(ph, g, cost, st2);
  if (done && kind == kCompton) ed = compton_energy(s, ph, eps);
  if (done) trials = 0u;
  return done;
}

// The dose kernel's part of a slot: the history's voxel list.
template <typename real>
struct VoxelList {
  uint32_t vox[kHistList];
  alignas(16) real acc[kHistList];
};
template <>
struct VoxelList<double> {
  uint32_t vox[kHistList];
  alignas(16) double acc[kHistList];
  uint4 pad;
};
template <typename real>
using DoseSlot = PhotonSlot<real, VoxelList<real>>;
// ... with the dose per entry beside it, for a dose grid that scores both; the
// two lists have the same voxels
template <typename real>
struct VoxelListDose {
  uint32_t vox[kHistList];
  alignas(16) real acc[kHistList];
  alignas(16) real dose[kHistList];
};
template <>
struct VoxelListDose<double> {
  uint32_t vox[kHistList];
  alignas(16) double acc[kHistList];
  alignas(16) double dose[kHistList];
  uint4 pad;
};
template <typename real>
using GridSlot = PhotonSlot<real, VoxelListDose<real>>;
// ... and, with the track-length estimator, its walk through the voxels: next
// boundary per axis and path so far, boundary spacing per axis and drawn path,
// voxel per axis and boundaries crossed.
template <typename real>
struct TlePad {};
template <>
struct TlePad<float> {
  uint4 pad;
};
template <typename real>
struct VoxelWalkList : TlePad<real> {
  uint32_t vox[kHistList];
  alignas(16) real acc[kHistList];
  Real4<real> tn, td;
  int4 it;
};
template <typename real>
using TleSlot = PhotonSlot<real, VoxelWalkList<real>>;
static_assert(sizeof(DoseSlot<float>) % 32 == 16 && sizeof(DoseSlot<double>) % 32 == 16 &&
                  sizeof(TleSlot<float>) % 32 == 16 && sizeof(TleSlot<double>) % 32 == 16 &&
                  sizeof(GridSlot<float>) % 32 == 16 && sizeof(GridSlot<double>) % 32 == 16,
              "odd 16-byte stride");
static_assert(kHistList == 8, "list_deposit reads the voxels as two 16-byte words");

// A history's voxel list in its slot (the entries of HistList, in their order).
// list_deposit(): all voxels are compared at once - a loop over the entries makes
// the warp wait for its longest list.  Returns the entry (-1: nothing to score);
// flush(k): entry k of a full list into the tallies.
template <typename real, typename List, typename Flush>
__device__ __forceinline__ int list_deposit(List &S, int &n, uint32_t v, real e, unsigned int &n_dep,
                                            unsigned int &n_entries, unsigned int &n_over, Flush &&flush) {
  if (!(e > R<real>(0))) return -1;
  ++n_dep;
  const uint4 a = *reinterpret_cast<const uint4 *>(S.vox), b = *reinterpret_cast<const uint4 *>(S.vox + 4);
  const uint32_t u[kHistList] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  int at = n;
#pragma unroll
  for (int k = kHistList - 1; k >= 0; --k)
    if (k < n && u[k] == v) at = k;
  if (at < n) {
    S.acc[at] = S.acc[at] + e;
    return at;
  }
  if (n == kHistList) {
    ++n_over;
    n_entries += kHistList;
#pragma unroll 1
    for (int k = 0; k < kHistList; ++k) flush(k);
    n = at = 0;
  }
  S.vox[at] = v;
  S.acc[at] = e;
  n = at + 1;
  return at;
}

// The lists of the warp's ended histories (`n` entries of the lane's slot
// `slot`) into the tallies: the entries are dealt over the lanes, one each -
// about 1.5 per history, but the longest of 32 lists has 4 or 5.  ids: 32 *
// kHistList numbers of the warp's own.  flush(slot, k): its entry k.
template <typename Slot, typename Flush>
__device__ __forceinline__ void lists_flush(const Slot *slots, int slot, int n, uint16_t *ids, unsigned lane,
                                            Flush &&flush, unsigned int &n_entries) {
  unsigned end = (unsigned)n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= (unsigned)o) end += x;
  }
  const unsigned total = __shfl_sync(0xffffffffu, end, 31);
  uint16_t *p = ids + (end - (unsigned)n);
#pragma unroll
  for (int k = 0; k < kHistList; ++k)
    if (k < n) p[k] = (uint16_t)(slot * kHistList + k);
  __syncwarp();
#pragma unroll 1
  for (unsigned i = lane; i < total; i += 32u) {
    const unsigned id = ids[i];
    flush(slots[id / kHistList], id % kHistList);
  }
  n_entries += (unsigned)n;
  __syncwarp();
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long x) {
  unsigned long long r = __reduce_add_sync(0xffffffffu, (unsigned)x & 0xffffffu);
  r += (unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(x >> 24) & 0xffffffu) << 24;
  return r + ((unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(x >> 48)) << 48);
}

// The first n entries of each lane's list into the tally, entry by entry;
// entries of the voxel that the first such lane holds are summed first and added
// once when they are several.  The photons of a narrow beam cross the same voxels in the
// same rounds, and their atomics otherwise queue at a few L2 slices.
constexpr int kSameVoxel = 3;
template <typename real, typename List>
__device__ __forceinline__ void lists_flush_same(const List &S, int n, const Tally<real> &t, unsigned lane) {
#pragma unroll 1
  for (int k = 0;; ++k) {
    const bool has = k < n;
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (m == 0u) break;
    const int first = __ffs(m) - 1;
    const uint32_t v = S.vox[min(k, kHistList - 1)];
    const unsigned long long q = has ? (unsigned long long)to_fixed(S.acc[k]) : 0ull;
    const uint32_t v0 = __shfl_sync(0xffffffffu, v, first);
    bool mine = has && v == v0;
    const unsigned same = __ballot_sync(0xffffffffu, mine);
    unsigned long long e = q, lo = (q * q) & 0xffffffffull, hi = (__umul64hi(q, q) << 32) | ((q * q) >> 32);
    if (__popc(same) >= kSameVoxel) {
      const unsigned long long se = warp_sum(mine ? e : 0ull);
      const unsigned long long sl = warp_sum(mine ? lo : 0ull), sh = warp_sum(mine ? hi : 0ull);
      if ((int)lane == first) {
        e = se;
        lo = sl;
        hi = sh;
        mine = false;
      }
    } else {
      mine = false;
    }
    if (has && !mine) {
      atomicAdd(&t.acc_e[v], e);
      if (t.acc_e2) {
        atomicAdd(&t.acc_e2[2 * (size_t)v], lo);
        atomicAdd(&t.acc_e2[2 * (size_t)v + 1], hi);
      }
    }
  }
}

// Boundaries a walk of the track-length estimator crosses in one round: their
// label loads are in flight together, but a path's last round leaves lanes idle
// (2 / 3 / 4 / 5 / 6 / 8 boundaries: 9.5 / 7.8 / 6.9 / 7.1 / 7.0 / 7.5 ms, the
// workload of k_transport_pool).
constexpr int kTleSteps = 4;
static_assert(kTleSteps <= kHistList, "the list holds what is left of a round after a flush");

template <typename real>
__device__ __forceinline__ void tle_store(VoxelWalkList<real> &X, const VoxelWalk<real> &w, real sd) {
  X.tn = Real4<real>{w.tn[0], w.tn[1], w.tn[2], w.tc};
  X.td = Real4<real>{w.td[0], w.td[1], w.td[2], sd};
  X.it = make_int4(w.i[0], w.i[1], w.i[2], w.k);
}

// One round of the estimator's walks (slot k of each lane, -1: none); the
// slot's next event.  The warp calls it together; a lane without a slot reads
// slot 0, which may never have held a photon, so nothing of it becomes an address.
template <typename real>
__device__ __forceinline__ int tle_walk(const Scene<real> &s, TleSlot<real> *slots, int k, unsigned lane,
                                        const Tally<real> &t, unsigned int &n_dep, unsigned int &n_ent,
                                        unsigned int &n_over) {
  TleSlot<real> &S = slots[max(k, 0)];
  const uint4 e = S.e;
  const Real4<real> b = S.b, tn = S.x.tn, td = S.x.td;
  const int4 it = S.x.it;
  VoxelWalk<real> w{{tn.x, tn.y, tn.z}, {td.x, td.y, td.z}, tn.w, {it.x, it.y, it.z}, it.w};
  const real d[3] = {b.x, b.y, b.z}, len = td.w < S.a.w ? td.w : S.a.w;
  EIdx<real> ei;
  ei.fe = S.c.z;
  ei.ie = k >= 0 ? (int)(real_bits(S.c.w) & 0xffffu) : 0;
  // the crossings, then their labels with all loads in flight, then the energies
  uint32_t v[kTleSteps];
  real ed[kTleSteps];
  bool more = k >= 0;
#pragma unroll
  for (int j = 0; j < kTleSteps; ++j) {
    v[j] = 0u;
    ed[j] = R<real>(0);
    if (more) more = w.step(s, d, len, v[j], ed[j]);
  }
  int m[kTleSteps];
#pragma unroll
  for (int j = 0; j < kTleSteps; ++j) m[j] = (int)__ldg(s.labels + v[j]);
  int last = -1;
  real mu_e = R<real>(0);
#pragma unroll
  for (int j = 0; j < kTleSteps; ++j) {
    if (m[j] != last) {
      last = m[j];
      real mu = interp_row(s.muen + (size_t)s.mat_comp[last] * s.n_e, ei);
      mu = s.mat_rho[last] * mu;
      mu_e = b.w * mu;
    }
    ed[j] = ed[j] > R<real>(0) ? mu_e * ed[j] : R<real>(0);
  }
  // into the list: a walk never comes back to a voxel, so only the entries from
  // before this round can be a crossing's voxel, and none once the list is flushed
  int n = (int)((e.z >> kSlList) & 15u), n_old = n;
  const uint4 ua = *reinterpret_cast<const uint4 *>(S.x.vox), ub = *reinterpret_cast<const uint4 *>(S.x.vox + 4);
  const uint32_t u[kHistList] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
  bool full = false;
#pragma unroll
  for (int j = 0; j < kTleSteps; ++j) {
    if (ed[j] > R<real>(0) && !full) {
      int at = n;
#pragma unroll
      for (int q = 0; q < kHistList; ++q)
        if (q < n_old && u[q] == v[j]) at = q;
      if (at == kHistList) {
        full = true;
      } else {
        const bool add = at == n;
        S.x.vox[at] = v[j];
        S.x.acc[at] = add ? ed[j] : S.x.acc[at] + ed[j];
        n += add ? 1 : 0;
        ++n_dep;
        ed[j] = R<real>(0);
      }
    }
  }
  __syncwarp();
  if (__any_sync(0xffffffffu, full)) {
    lists_flush_same(S.x, full ? n : 0, t, lane);
    if (full) {
      ++n_over;
      n_ent += kHistList;
      n = 0;
#pragma unroll
      for (int j = 0; j < kTleSteps; ++j)
        if (ed[j] > R<real>(0)) {
          S.x.vox[n] = v[j];
          S.x.acc[n] = ed[j];
          ++n;
          ++n_dep;
        }
    }
  }
  if (k < 0) return kQNone;
  S.x.tn = Real4<real>{w.tn[0], w.tn[1], w.tn[2], w.tc};
  S.x.it = make_int4(w.i[0], w.i[1], w.i[2], w.k);
  S.e.z = (e.z & ~(15u << kSlList)) | ((uint32_t)n << kSlList);
  return more ? kQWalk : kQFly;
}

}  // namespace gg
