// gg_internal.h - declarations shared by the host API and the kernel translation units.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace gg {

// cudaFuncSetAttribute applies to the current device only: `done` remembers,
// one bit per device ordinal (< 64), on which devices a kernel's dynamic
// shared-memory limit has been raised: to `bytes`, or to what the block's
// opt-in limit leaves beside the kernel's static shared memory if less.
template <typename K>
inline cudaError_t configure_smem(K kernel, int bytes, unsigned long long &done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
  if (bit && (done & bit)) return cudaSuccess;
  int optin = 0;
  cudaFuncAttributes fa;
  if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  if ((e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess) return e;
  const int room = optin - (int)fa.sharedSizeBytes;
  if (room < bytes) bytes = room;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done |= bit;
  return e;
}

// Launch of a kernel that may start (overlap) while the stream's previous kernel ends: it
// calls cudaGridDependencySynchronize() before it touches that kernel's data.
template <typename... P, typename... A>
inline cudaError_t launch_overlapped(bool overlap, void (*kernel)(P...), int grid, int block, size_t smem,
                                     cudaStream_t st, A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, args...);
}

template <typename real>
struct Scene;

// Arguments of one transport launch (one tally batch).
struct KernelArgs {
  uint64_t seed;
  uint64_t h_begin, h_end;          // histories [h_begin, h_end)
  unsigned long long *next;         // claim counter, zero at launch
  unsigned long long *acc_e;        // per-voxel fixed-point edep of this batch
  unsigned long long *acc_e2;       // per-voxel fixed-point edep^2 (or null)
  unsigned long long *counters;     // GG_N_COUNTERS slots
  unsigned int *status;             // OR of error codes raised by the kernel
  int chunk;                        // histories claimed per warp refill
  void *records;                    // primary records of the batch (k_generate -> transport)
  size_t rec_cap;                   // records capacity (histories per batch)
  uint64_t rec_first;               // history of record 0 (<= h_begin; a SPECT pass can start later)
  int refill_min;                   // lanes that must wait before a refill phase (SPECT head stage)
  int interact_min;                 // pending collisions that trigger its interaction phase
  unsigned long long *acc_d;        // dose grid: fixed-point sum(edep * rho_min / rho) (or null)
  unsigned long long *acc_d2;       // its history-by-history squares (or null)
  void *slot_scratch;               // pooled kernels: PoolPlan::scratch bytes
};

// Bit of the kernel status word set when a stage queue overflowed (the low
// bits carry the source stage's GG_ERR_* code).
constexpr unsigned int kStatusQueueOverflow = 0x100u;
// Bit set when a bounded wait of a tensor-core kernel ran out (the kernel
// stopped early and freed its tensor memory).
constexpr unsigned int kStatusWaitTimeout = 0x200u;

// Queues of one SPECT stage launch (see gg_spect.cu).
struct StageArgs {
  void *in_q;                      // input queue (phantom stage: null = the batch's primary records)
  const unsigned long long *in_n;  // input queue length
  void *out_q;                     // output queue
  unsigned long long *out_n;       // output queue length (appended to)
  size_t q_cap;                    // capacity of each queue (entries)
  // scatter splitting: requests of the phantom stage for the split kernel
  // (Compton from the front, Rayleigh from the back of one buffer)
  void *split_q;
  unsigned long long *split_n;     // [Compton requests, Rayleigh requests]
  size_t split_cap;
};

// One launch of the ARF training-row generator (see gg_arf.cu).
constexpr int kArfBlock = 256;

struct ArfArgs {
  uint64_t seed, first, n;        // samples [first, first + n), Philox stream 1
  double e_min, e_max, cos_theta_max, half_extent[2], russian_roulette;
  int theta_uniform;              // theta = u theta_max instead of cos(theta) uniform
  double theta_max_turn;          // acos(cos_theta_max) / (2 pi)
  float4 *stage;                  // [n] row per sample (w = -1: dropped)
  unsigned long long *next;       // work counter
  unsigned int *block_count;      // [blocks] kept rows per block of kArfBlock samples
  unsigned long long *block_off;  // [blocks] first output row of each block
  unsigned long long *counters;   // GG_N_COUNTERS slots
};

// One training step (or a prediction) of the ARF network (see gg_mlp.cu).
struct MlpTrainArgs {
  const float4 *rows;            // (E, theta, phi, class) rows
  uint64_t row0, n_rows;         // tile t reads rows (row0 + 128 t + r) % n_rows
  const float *params;           // FP32 parameters
  const __nv_bfloat16 *wbf;      // BF16 copies of W2, W3, W4
  float *partial;                // [tiles][kNParams] gradient of each tile (param_of_partial order)
  float *loss_part;              // [tiles] loss sum of each tile
  float mean[3], inv_std[3];     // standardisation of (theta, phi, E)
  int n_classes;
  float inv_batch;               // 1 / rows in the step
  unsigned int *status;          // kStatusWaitTimeout when a tensor-core wait ran out
};

constexpr int kTrainRows = 128;  // rows per training tile (one CTA, MMA M)

struct MlpAdamArgs {
  const float *partial;
  int n_tiles;
  float *params;
  __nv_bfloat16 *wbf;
  float *m, *v;                  // Adam moments (param_of_partial order)
  float *grad_out;               // summed gradient (or null)
  float lr, beta1, beta2, eps;   // lr = 0: gradient only, no update
  float c1, c2;                  // 1 / (1 - beta1^t), 1 / (1 - beta2^t)
  const float *loss_part;        // [n_tiles] tile loss sums, added to *loss_acc (or null)
  double *loss_acc;
};

// One launch of the ARF stage of the SPECT wavefront (see gg_arf_stage.cu).
struct ArfStageArgs {
  void *in_q;                      // head queue of the phantom stage
  const unsigned long long *in_n;
  void *out_q;                     // fallback queue for the plain head stage
  unsigned long long *out_n;
  size_t q_cap;
  const float *params;             // network
  const __nv_bfloat16 *wbf;
  float mean[3], inv_std[3];
  int n_classes;
  float rr;                        // class-0 Russian-roulette factor of the training rows
  double e_min, e_max, cos_theta_max;  // trained domain
  double e_detect_min;             // lowest window edge: photons below reach no window
  double dc;                       // collimator face -> crystal plane, mm
  unsigned long long *proj;        // fixed-point window weights, 2^-32 units, projection layout
  unsigned long long *proj2;       // their squares: (low 32 bits, rest) per pixel, 2^-64 / 2^-32 MeV^2 units
  unsigned long long *counters;
  unsigned int *status;
  unsigned long long *claim;       // chunk claim counter, zero at launch
};

size_t mlp_train_smem_bytes();
cudaError_t launch_mlp_train(const MlpTrainArgs &a, int n_tiles, bool overlap, cudaStream_t st);
cudaError_t launch_mlp_adam(const MlpAdamArgs &a, bool overlap, cudaStream_t st);
// *bad = number of the first invalid training row, if below its value
cudaError_t launch_check_rows(const float4 *rows, uint64_t n, int n_classes, unsigned long long *bad, int n_sm,
                              cudaStream_t st);
cudaError_t launch_mlp_to_bf16(const float *params, __nv_bfloat16 *wbf, cudaStream_t st);
size_t mlp_tc_smem_bytes();
cudaError_t launch_mlp_predict(const MlpTrainArgs &a, float *out, uint64_t n, int grid, unsigned int *status,
                               cudaStream_t st);
template <typename real>
cudaError_t launch_spect_arf(const Scene<real> &s, const ArfStageArgs &a, int grid, cudaStream_t st);

constexpr int kHistList = 8;     // entries of a history's voxel list
constexpr int kBlock = 256;      // most threads per block of the transport kernels
constexpr int kTransportSmemMax = 200 * 1024;  // dynamic shared memory of a transport block

// Shared memory of the transport kernels' tables: sigma rows, majorant, density
// and composition index per material, 16-byte aligned.
template <typename real>
__host__ __device__ inline size_t transport_smem_bytes(int n_comp, int n_e, int n_mat) {
  size_t b = sizeof(real) * ((size_t)n_comp * n_e + n_e + n_mat) + sizeof(int) * (size_t)n_mat;
  return (b + 15) & ~(size_t)15;
}

// Shared memory of `lists` per-history voxel lists of `threads` histories: the
// room that the largest tables leave to a pooled kernel's photons.
template <typename real>
__host__ __device__ constexpr size_t hist_list_bytes(int lists, int threads = kBlock) {
  return (size_t)lists * kHistList * (size_t)threads * (sizeof(uint32_t) + sizeof(real));
}
// Launch shape of a pooled transport kernel (gg_pool.cuh).
struct PoolPlan {
  int grid, block, gangs, slots;  // blocks, threads and gangs per block, photon slots per gang
  int gang_threads;               // (the last gang may have fewer)
  size_t smem, scratch;           // dynamic shared memory; global scratch (KernelArgs::slot_scratch)
};
// Threads of a block (one block per SM), warps of a full block's gang, most gangs
// of a block, entries of an event queue's ring (more than a gang's slots).  Measured on the 256 x 256 x 160 CT,
// 1e8 histories (transport ms): gangs of 2 / 3 / 4 / 6 / 12 warps of 24: 37.9 /
// - / 33.5 / 32.5 / 34.6 (small gangs fetch more instructions, large ones wait
// at their barrier); 16 / 18 / 20 / 24 warps in gangs of 4 / 3 / 4 / 4: 32.4 /
// 30.4 / 30.4 / 33.5 (more warps leave fewer slots each); 20 warps in gangs of
// 4 / 5: 30.7 / 30.8, the phantom stage of 3e7 decays 13.0 / 12.5, the track-length
// estimator 6.7 / 6.5 (24 in gangs of 4: 14.9, 7.2).  FP64, 128 x 128 x 80
// CT, 1e6 histories: 8 / 9 / 12 / 16 warps in gangs of 4 / 3 / 4 / 8: 4.64 /
// 4.22 / 4.86 / 5.16 ms (FP64 units bound it: full rounds count, not warps).
template <typename real>
struct PoolShape {
  static constexpr int kBlock = 640, kGang = 5, kGangs = 5, kRing = 512;
};
template <>
struct PoolShape<double> {
  static constexpr int kBlock = 288, kGang = 3, kGangs = 3, kRing = 512;
};
// (a block has 16 named barriers: number 0 for the block, one for each gang)
static_assert(PoolShape<float>::kGangs <= 15 && PoolShape<double>::kGangs <= 15, "more gangs than named barriers");
// static shared memory of a pooled kernel with as many event queues, at most
template <typename real>
__host__ __device__ constexpr int pool_static(int queues) {
  using P = PoolShape<real>;
  return 1024 + 16 * P::kBlock + P::kGangs * (2 * queues * P::kRing + (queues > 4 ? 112 : 64));
}
// Launch shape of a pooled run: one block per SM.  More slots per thread keep
// the rounds full, so they take all shared memory beside the tables, but no
// more than the run has histories for.  blocks: of the options, resident blocks
// per SM of 256 threads each, 0 for the kernel's register budget; as with the
// register budgets of the kernels that have several, 1 stands for 2 (1e7
// histories, 128 x 128 x 80 CT, 256 / 512 / 640 threads: 6.16 / 4.16 / 3.95 ms).
// The options' block_size means nothing here: 32 / 64 / 128 / 224 threads per SM
// take 36.6 / 19.3 / 10.3 / 6.8 ms.  slot_bytes, scratch_bytes: of one slot, shared
// and global.  False: the tables leave no room.
template <typename real>
inline bool pool_shape(int n_sm, size_t optin, size_t table_bytes, int blocks, uint64_t n_hist, size_t slot_bytes,
                       size_t scratch_bytes, int queues, PoolPlan *p) {
  using Shape = PoolShape<real>;
  constexpr int kGang = 32 * Shape::kGang;
  const uint64_t per_sm = (n_hist + n_sm - 1) / n_sm;
  int threads = Shape::kBlock;
  if (blocks > 0) threads = std::min(threads, 256 * std::max(std::min(blocks, 4), 2));
  threads = (int)std::min<uint64_t>(threads, (per_sm + 31) / 32 * 32);
  const size_t fixed = pool_static<real>(queues) + table_bytes;
  const int room = optin > fixed ? (int)((optin - fixed) / slot_bytes) : 0;
  while (threads > kGang && room < threads) threads -= kGang;  // (large tables: fewer gangs)
  // a small run's block has as many gangs as may be: a photon then waits for fewer others'
  // events (2e4 / 4e4 / 6e4 histories, us, gangs of kGang: 64^3 water 94 / 100 / 109 -> 85 / 94 /
  // 96, 128 x 128 x 80 CT 219 / 233 / 244 -> 189 / 211 / 229; from a full block on the same)
  const int gang = room < threads || threads == Shape::kBlock
                       ? kGang
                       : (threads + 32 * Shape::kGangs - 1) / (32 * Shape::kGangs) * 32;
  const int gangs = (threads + gang - 1) / gang;
  const int most = std::min(room / gangs, Shape::kRing - 32) / 8 * 8;
  if (most < 8) return false;
  const uint64_t share = std::max<uint64_t>((per_sm + gangs - 1) / gangs, 32);
  p->grid = n_sm;
  p->block = threads;
  p->gangs = gangs;
  p->gang_threads = gang;
  p->slots = (int)std::min<uint64_t>(most, (share + 7) / 8 * 8);
  p->smem = slot_bytes * p->slots * gangs + table_bytes;
  p->scratch = (size_t)p->grid * gangs * p->slots * scratch_bytes;
  return true;
}
// Photon slots of a pooled run of n histories, at most: one for each, an SM's histories
// rounded up to warps (a gang has 32 slots at least) or its gangs' shares to 8.
template <typename real>
constexpr size_t pool_slots_most(uint64_t n, int n_sm) {
  return (size_t)n + (size_t)n_sm * (1 + std::max(31, 8 * PoolShape<real>::kGangs));
}
template <typename real>
cudaError_t pool_plan(int device, size_t table_bytes, int blocks, uint64_t n_hist, size_t slot_bytes,
                      size_t scratch_bytes, int queues, PoolPlan *p);
// Histories a gang claims at a time: an even share of a small run, so that all gangs
// work on it (10 / 1000 / 5000 histories, 128 x 128 x 80 CT: 0.156 / 0.211 / 0.231 ms with at
// least 32, 0.146 / 0.194 / 0.213 so), else the per-warp chunk of the options for each of its
// warps, and then no less than a warp's lanes.
inline int pool_chunk(const PoolPlan &p, int chunk, uint64_t n_hist) {
  const uint64_t gangs = (uint64_t)p.grid * p.gangs, share = (n_hist + gangs - 1) / gangs;
  const uint64_t warps = (uint64_t)std::max(p.block / 32 / p.gangs, 1);
  const uint64_t most = std::max<uint64_t>(32, warps * (uint64_t)std::min(std::max(chunk, 1), 1 << 20));
  return (int)std::max<uint64_t>(1, std::min(share, most));
}
// Shared memory of a dose slot (tle: with the track-length estimator; two: a
// dose grid that scores edep and dose); its global scratch.
template <typename real>
size_t dose_slot_bytes(bool tle, bool two);
template <typename real>
size_t slot_scratch_bytes();
// Rows of p.n samples appended to rows[*total ...] (capacity rows); *total advances on the device.
template <typename real>
cudaError_t launch_arf_dataset(const Scene<real> &s, const ArfArgs &p, int n_sm, float4 *rows, uint64_t capacity,
                               unsigned long long *total, cudaStream_t st);
template <typename real>
size_t queue_bytes(size_t cap);
// Phantom and head stages of the SPECT wavefront (gg_spect.cu)
template <typename real>
cudaError_t launch_spect_phantom(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, const PoolPlan &p,
                                 int n_sm, cudaStream_t st);
template <typename real>
size_t phantom_slot_bytes();
template <typename real>
cudaError_t launch_spect_head(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int grid, int block,
                              size_t smem, int minb, cudaStream_t st);
template <typename real>
cudaError_t spect_head_occupancy(int block, size_t smem, int minb, int *blocks_per_sm);
// Copies of scatter splitting (gg_spect.cu): the split requests of q.split_q
// into the walk queue (q.out_q / q.out_n); does nothing when the requests
// overflowed the buffer.
template <typename real>
cudaError_t launch_spect_split(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int n_sm,
                               cudaStream_t st);
template <typename real>
size_t split_bytes(size_t cap);
// Free flights of the copies the split kernel queued (q.in_q / q.in_n) into
// the head queue (q.out_q / q.out_n).
template <typename real>
cudaError_t launch_spect_walk(const Scene<real> &s, const KernelArgs &a, const StageArgs &q, int block, size_t smem,
                              int n_sm, cudaStream_t st);
// A projection tally (counts; fixed-point weights; their squares, two words per pixel) as FP64.
enum : int { kProjCounts = 0, kProjWeights = 1, kProjSquares = 2 };
cudaError_t launch_projection_f64(int kind, const unsigned long long *src, double *dst, size_t n, int n_sm,
                                  cudaStream_t st);
template <typename real>
size_t record_bytes(size_t cap);
template <typename real>
cudaError_t launch_generate(const Scene<real> &s, const KernelArgs &a, cudaStream_t st);
template <typename real>
cudaError_t launch_transport(const Scene<real> &s, const KernelArgs &a, const PoolPlan &p, cudaStream_t st);
// Compacted wavefront dose transport (gg_wavefront.cu): 256-thread blocks,
// dynamic shared memory = tables + photon slots.
template <typename real>
size_t wavefront_smem_bytes(int n_comp, int n_e, int n_mat);
template <typename real>
cudaError_t launch_wavefront(const Scene<real> &s, const KernelArgs &a, int grid, size_t smem, int minb,
                             cudaStream_t st);
template <typename real>
cudaError_t wavefront_occupancy(size_t smem, int minb, int *blocks_per_sm);
// image += fixed point * 2^-32 * scale (squares: * scale^2), then clears the fixed-point sums
cudaError_t launch_flush(unsigned long long *acc_e, unsigned long long *acc_e2, double *edep, double *edep2,
                         size_t n, int grid, cudaStream_t st, double scale = 1.0);

}  // namespace gg
