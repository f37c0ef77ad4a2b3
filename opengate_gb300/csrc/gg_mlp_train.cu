// gg_mlp_train.cu - one training step of the ARF network on the 5th-generation
// tensor cores.
//
// Same network, loss and storage points as the inference kernels (garf ARF
// model, opengate/actors/arfactors.py:349-415; softmax cross-entropy on the
// (E, theta, phi, class) rows of GateARFTrainingDatasetActor).  One CTA (four
// warpgroups) takes a tile of 128 rows.
//
//   forward: layer 1 on the CUDA cores; layers 2-4 as tcgen05.mma (M 128,
//     K 16 per instruction) from BF16 K-major operands into TMEM, epilogue per
//     thread (bias, ReLU, BF16) writing the next A operand [row][unit] and,
//     for H1 and H2, the transposed copy [unit][row]; ReLU masks stay in
//     registers;
//   output: softmax, loss, dL/dlogits = (p - onehot) / B in BF16 [row][class];
//   backward, per hidden layer l (dZ = BF16 gradient at the layer's output):
//     dW_l = dZ^T H_{l-1}: A = dZ^T [unit][row], B = H_{l-1}^T [unit][row],
//     dH_{l-1} = dZ W_l: A = dZ [row][unit], B = W_l^T (a bulk-loaded copy),
//     both issued back to back into two TMEM column ranges, one commit;
//     dW_l read back lane by lane into the tile's partial gradient; biases
//     and the small output / input layers on the CUDA cores.
// The per-tile gradients are summed in tile order by k_mlp_adam (gg_mlp.cu).
// Every mbarrier wait is bounded; a wait that runs out sets kStatusWaitTimeout
// and the tile stops (its tensor memory is freed).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_internal.h"
#include "gg_mlp.cuh"
#include "gg_mlp_tc.cuh"
#include "gg_tc.cuh"

namespace gg {

constexpr int kTrGroups = 4;                           // warpgroups per tile
constexpr int kTrThreads = kTrainRows * kTrGroups;
constexpr int kTrBytesDz4 = kTrainRows * kOutPad * 2;  // dL/dlogits, [row][class], K = 16
// Activations and their transposes: core matrices adjacent along K lie 144 bytes
// apart (not 128), so the lanes of a warp that write or read one column of 32
// rows reach 32 banks instead of four lanes each.
constexpr uint32_t kTrLbo = kTcLbo + 16u;
constexpr uint32_t kTrSbo = (kHid / 8) * kTrLbo;
constexpr int kTrBytesAct = (int)(kTrainRows / 8 * kTrSbo);

__host__ __device__ constexpr uint32_t tr_offset(int r, int k) {
  return (uint32_t)(r >> 3) * kTrSbo + (uint32_t)(k >> 3) * kTrLbo + (uint32_t)(r & 7) * 16u + (uint32_t)(k & 7) * 2u;
}

constexpr int kMaxClasses = 9;  // energy windows + 1

struct TrainSmem {
  alignas(1024) uint8_t w2[kTcBytesHid];  // forward W2 [out][in]; backward W2^T [in][out]
  alignas(1024) uint8_t w3[kTcBytesHid];  // forward W3; backward W3^T
  alignas(1024) uint8_t w4[kTcBytesOut];  // forward W4 [16][128]; backward W4^T [128][16]
  alignas(128) uint8_t act[kTrBytesAct];  // [row][unit]: H1, H2, H3, then dZ3, dZ2
  alignas(128) uint8_t h1t[kTrBytesAct];  // H1^T [unit][row]
  alignas(128) uint8_t h2t[kTrBytesAct];  // H2^T
  alignas(128) uint8_t dzt[kTrBytesAct];  // dZ^T [unit][row] of the current layer
  alignas(128) uint8_t dz4[kTrBytesDz4];  // dL/dlogits [row][class]
  float4 w1[kHid];                        // layer 1: weights of the unit, bias
  float b2[kHid], b3[kHid], b4[kOutPad];
  alignas(16) float x[3][kTrainRows];     // inputs
  alignas(16) float dz4f[kMaxClasses][kTrainRows];  // dL/dlogits as stored, FP32
  alignas(16) float loss[kTrainRows];
  uint64_t mbar_mma, mbar_load;
  uint32_t tmem_base;
};
static_assert(sizeof(TrainSmem) <= 227 * 1024, "one tile fits an SM's shared memory");

constexpr uint32_t kTrCols = 256;  // TMEM: columns [0, 128) dW / forward, [128, 256) dH

__device__ __forceinline__ uint32_t bf2_pack(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}

// Writes unit values v[0..31] (units col0 ..) of row r: BF16 into the A operand
// [row][unit] (16-byte stores) and, when t != nullptr, into the transposed
// operand [unit][row] (one element per unit).
__device__ __forceinline__ void tr_store32(uint8_t *act, uint8_t *t, int r, int col0, const float (&v)[32]) {
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = bf2_pack(v[2 * i], v[2 * i + 1]);
  if (act) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<uint4 *>(act + tr_offset(r, col0 + 8 * c)) =
          make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
  }
  if (t) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      *reinterpret_cast<uint16_t *>(t + tr_offset(col0 + i, r)) = (uint16_t)(i & 1 ? w[i / 2] >> 16 : w[i / 2]);
  }
}

// Sum over the tile's rows of row j of a transposed operand [unit][row].
__device__ __forceinline__ float tr_row_sum(const uint8_t *t, int j) {
  float s = 0.0f;
#pragma unroll 4
  for (int c = 0; c < kTrainRows / 8; ++c) {
    const uint4 q = *reinterpret_cast<const uint4 *>(t + tr_offset(j, 8 * c));
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      s += f.x;
      s += f.y;
    }
  }
  return s;
}

// Issues the MMAs of D (+)= A B^T, K = kk in steps of 16, into d_tmem (no
// commit); lbo, sbo: the strides of each operand's core matrices.
__device__ __forceinline__ void tr_mma(uint32_t d_tmem, const uint8_t *a, uint32_t a_lbo, uint32_t a_sbo,
                                       const uint8_t *b, uint32_t b_lbo, uint32_t b_sbo, int n, int kk) {
  const uint32_t a0 = tc_smem(a), b0 = tc_smem(b), idesc = tc_idesc_bf16(kTrainRows, n);
  for (int ks = 0; ks < kk / 16; ++ks)
    tc_mma_bf16(d_tmem, tc_desc(a0 + 2u * a_lbo * ks, a_lbo, a_sbo), tc_desc(b0 + 2u * b_lbo * ks, b_lbo, b_sbo), idesc,
                ks > 0 ? 1u : 0u);
}

// Waits for MMA batch `phase` of the CTA; the result is the same for every thread.
__device__ __forceinline__ bool tr_wait(TrainSmem &sm, uint32_t &phase) {
  bool ok = mbar_wait(&sm.mbar_mma, phase & 1u, kTcWaitLimit);
  if (!ok) mbar_wait(&sm.mbar_mma, phase & 1u, kTcWaitLimit);  // let MMAs in flight finish
  ++phase;
  ok = __syncthreads_and(ok) != 0;
  tc_fence_after();
  return ok;
}

// Generic-proxy shared-memory writes visible to the tensor core, TMEM reads
// ordered, all threads past this point; then thread 0 may issue MMAs.
__device__ __forceinline__ void tr_publish() {
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
}


// Four warpgroups share a tile: thread t owns row (forward) or unit (gradient
// read-back) t % 128 and the 32 columns 32 g .. of its group g = t / 128, since a
// single warpgroup leaves one warp per scheduler and every epilogue a serial
// chain.  Sums over rows keep their order (one thread per sum).
// Latency bound: a step of 64 tiles (this kernel and the optimiser's) 49.1 -> 28.7
// us, with overlapped launches 23.8; 512 tiles 205 -> 109.
__global__ void __launch_bounds__(kTrThreads, 1) k_mlp_train(MlpTrainArgs a) {
  extern __shared__ __align__(1024) unsigned char tr_smem_raw[];
  TrainSmem &sm = *reinterpret_cast<TrainSmem *>(tr_smem_raw);
  const int r = threadIdx.x & (kTrainRows - 1);  // row (forward), unit (gradient read-back)
  const int g = threadIdx.x / kTrainRows, col0 = 32 * g;
  const int tile = blockIdx.x;
  float *part = a.partial + (size_t)tile * kNParams;
  const uint32_t tlane = (uint32_t)(32 * (r >> 5)) << 16;  // the warp's TMEM lane quarter

  // ---- set-up: mbarriers, inputs, TMEM; then forward weights (bulk copies) ----
  cudaTriggerProgrammaticLaunchCompletion();  // (the optimiser's kernel waits for this grid's end)
  if (threadIdx.x == 0) {
    mbar_init(&sm.mbar_mma, 1u);
    mbar_init(&sm.mbar_load, 1u);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const float4 row = a.rows[(a.row0 + (uint64_t)tile * kTrainRows + (uint64_t)r) % a.n_rows];
  const float x0 = (row.y - a.mean[0]) * a.inv_std[0];
  const float x1 = (row.z - a.mean[1]) * a.inv_std[1];
  const float x2 = (row.x - a.mean[2]) * a.inv_std[2];
  const int y = (int)row.w;
  if (g == 3) {
    sm.x[0][r] = x0;
    sm.x[1][r] = x1;
    sm.x[2][r] = x2;
  }
  if (threadIdx.x < 32) {
    tmem_alloc(&sm.tmem_base, kTrCols);
    tmem_relinquish();
  }
  __syncthreads();
  cudaGridDependencySynchronize();  // the previous step's parameters
  const __nv_bfloat16 *wtc = a.wbf, *wtt = a.wbf + kTcTBf;
  if (threadIdx.x == 0) {
    mbar_expect_tx(&sm.mbar_load, (uint32_t)(2 * kTcBytesHid + kTcBytesOut));
    bulk_load(sm.w2, wtc + kBfW2, (uint32_t)kTcBytesHid, &sm.mbar_load);
    bulk_load(sm.w3, wtc + kBfW3, (uint32_t)kTcBytesHid, &sm.mbar_load);
    bulk_load(sm.w4, wtc + kBfW4, (uint32_t)kTcBytesOut, &sm.mbar_load);
  }
  if (g == 0)
    sm.w1[r] = make_float4(a.params[kOffW1 + 3 * r], a.params[kOffW1 + 3 * r + 1], a.params[kOffW1 + 3 * r + 2],
                           a.params[kOffB1 + r]);
  if (g == 1) sm.b2[r] = a.params[kOffB2 + r];
  if (g == 2) sm.b3[r] = a.params[kOffB3 + r];
  if (g == 3 && r < kOutPad) sm.b4[r] = a.params[kOffB4 + r];
  __syncthreads();  // w1
  uint32_t mask1 = 0, mask2 = 0, mask3 = 0;  // ReLU masks of the thread's 32 columns
  // ---- layer 1 (CUDA cores): H1 -> act, H1^T -> h1t; the weights arrive meanwhile ----
  {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float4 w = sm.w1[col0 + i];
      float z = w.w;
      z = fmaf(w.x, x0, z);
      z = fmaf(w.y, x1, z);
      z = fmaf(w.z, x2, z);
      const bool on = z > 0.0f;
      v[i] = on ? z : 0.0f;
      if (on) mask1 |= 1u << i;
    }
    tr_store32(sm.act, sm.h1t, r, col0, v);
  }
  bool ok = mbar_wait(&sm.mbar_load, 0u, kTcWaitLimit);
  if (!ok) mbar_wait(&sm.mbar_load, 0u, kTcWaitLimit);
  tc_fence_before();
  ok = __syncthreads_and(ok) != 0;
  tc_fence_after();
  const uint32_t d_a = sm.tmem_base, d_b = sm.tmem_base + 128u;
  const uint32_t kSboHid = tc_sbo(kHid), kSboOut = tc_sbo(kOutPad);
  uint32_t phase = 0;

  if (ok) {
    // ---- layers 2, 3 (tensor cores) ----
#pragma unroll 1
    for (int layer = 0; layer < 2 && ok; ++layer) {
      tr_publish();
      if (threadIdx.x == 0) {
        tc_fence_after();
        tr_mma(d_a, sm.act, kTrLbo, kTrSbo, layer == 0 ? sm.w2 : sm.w3, kTcLbo, kSboHid, kHid, kHid);
        tc_commit(&sm.mbar_mma);
      }
      ok = tr_wait(sm, phase);
      if (!ok) break;
      const float *b = (layer == 0 ? sm.b2 : sm.b3) + col0;
      uint32_t mask = 0;
      float v[32];
      tmem_ld32(d_a + tlane + (uint32_t)col0, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float z = v[i] + b[i];
        const bool on = z > 0.0f;
        v[i] = on ? z : 0.0f;
        if (on) mask |= 1u << i;
      }
      tr_store32(sm.act, layer == 0 ? sm.h2t : nullptr, r, col0, v);
      if (layer == 0) mask2 = mask;
      else mask3 = mask;
    }
  }
  if (ok) {
    // ---- output layer, softmax, loss, dL/dlogits ----
    tr_publish();
    if (threadIdx.x == 0) {
      tc_fence_after();
      tr_mma(d_a, sm.act, kTrLbo, kTrSbo, sm.w4, kTcLbo, kSboHid, kOutPad, kHid);
      tc_commit(&sm.mbar_mma);
    }
    ok = tr_wait(sm, phase);
  }
  if (ok) {
    // the backward weight copies replace the forward ones (all forward MMAs are complete)
    if (threadIdx.x == kTrainRows) {
      mbar_expect_tx(&sm.mbar_load, (uint32_t)(2 * kTcBytesHid + kTcBytesOut));
      bulk_load(sm.w4, wtt + kBfW4, (uint32_t)kTcBytesOut, &sm.mbar_load);
      bulk_load(sm.w3, wtt + kBfW3, (uint32_t)kTcBytesHid, &sm.mbar_load);
      bulk_load(sm.w2, wtt + kBfW2, (uint32_t)kTcBytesHid, &sm.mbar_load);
    }
    if (g == 0) {
      float p[16];
      {
        float v[16];
        tmem_ld16(d_a + tlane, v);
#pragma unroll
        for (int c = 0; c < 16; ++c) p[c] = v[c] + sm.b4[c];
      }
      tc_softmax(p, a.n_classes);
      float py = 1.0f;
#pragma unroll
      for (int c = 0; c < 16; ++c)
        if (c == y) py = p[c];
      sm.loss[r] = -logf(fmaxf(py, 1e-30f));
      uint32_t w[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float g0 = 2 * c < a.n_classes ? (p[2 * c] - (2 * c == y ? 1.0f : 0.0f)) * a.inv_batch : 0.0f;
        float g1 = 2 * c + 1 < a.n_classes ? (p[2 * c + 1] - (2 * c + 1 == y ? 1.0f : 0.0f)) * a.inv_batch : 0.0f;
        w[c] = bf2_pack(g0, g1);
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[c]));
        if (2 * c < kMaxClasses) sm.dz4f[2 * c][r] = f.x;
        if (2 * c + 1 < kMaxClasses) sm.dz4f[2 * c + 1][r] = f.y;
      }
      *reinterpret_cast<uint4 *>(sm.dz4 + tc_offset(r, 0, kOutPad)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4 *>(sm.dz4 + tc_offset(r, 8, kOutPad)) = make_uint4(w[4], w[5], w[6], w[7]);
    }
    ok = mbar_wait(&sm.mbar_load, 1u, kTcWaitLimit);
    if (!ok) mbar_wait(&sm.mbar_load, 1u, kTcWaitLimit);
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok) != 0;
  }
  if (ok) {
    // ---- dH3 = dL W4 (K = 16), while the output layer's gradients run on the CUDA cores ----
    if (threadIdx.x == 0) {
      tc_fence_after();
      tr_mma(d_b, sm.dz4, kTcLbo, kSboOut, sm.w4, kTcLbo, kSboOut, kHid, kOutPad);
      tc_commit(&sm.mbar_mma);
    }
    // dW4[o][unit] = sum_row dz4[row][o] H3[row][unit] for the classes o = g, g + 4, ... (the
    // other outputs' gradients are zero); db4; the loss
    const uint8_t *hp = sm.act + tr_offset(0, r);
#pragma unroll 1
    for (int o = g; o < kOutPad; o += kTrGroups) {
      float sw = 0.0f;
      if (o < a.n_classes) {
        const float4 *dp = reinterpret_cast<const float4 *>(sm.dz4f[o]);
#pragma unroll
        for (int q = 0; q < kTrainRows; q += 4) {
          const float4 d = dp[q / 4];
          const float dz[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            sw = fmaf(dz[i], __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(hp + tr_offset(q + i, 0))), sw);
        }
      }
      part[kOffW4 + o * kHid + r] = sw;
    }
    if (threadIdx.x < kOutPad) {
      float sb = 0.0f;
      if (threadIdx.x < a.n_classes) {
#pragma unroll 8
        for (int q = 0; q < kTrainRows; ++q) sb += sm.dz4f[threadIdx.x][q];
      }
      part[kOffB4 + threadIdx.x] = sb;
    }
    if (threadIdx.x == kTrThreads - 32) {
      float s = 0.0f;
#pragma unroll 8
      for (int q = 0; q < kTrainRows; ++q) s += sm.loss[q];
      a.loss_part[tile] = s;
    }
    ok = tr_wait(sm, phase);  // (every thread is done with H3 in act)
  }
  // ---- hidden layers 3, 2: dZ = dH * mask -> act and dzt; dW = dZ^T H_in, dH_in = dZ W ----
#pragma unroll 1
  for (int layer = 0; layer < 2 && ok; ++layer) {
    const uint32_t mask = layer == 0 ? mask3 : mask2;
    {
      float v[32];
      tmem_ld32(d_b + tlane + (uint32_t)col0, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = (mask >> i) & 1u ? v[i] : 0.0f;
      tr_store32(sm.act, sm.dzt, r, col0, v);
    }
    tr_publish();
    if (threadIdx.x == 0) {
      tc_fence_after();
      // dH of the layer below, then dW
      tr_mma(d_b, sm.act, kTrLbo, kTrSbo, layer == 0 ? sm.w3 : sm.w2, kTcLbo, kSboHid, kHid, kHid);
      tr_mma(d_a, sm.dzt, kTrLbo, kTrSbo, layer == 0 ? sm.h2t : sm.h1t, kTrLbo, kTrSbo, kHid, kTrainRows);
      tc_commit(&sm.mbar_mma);
    }
    // db while the MMAs run
    const int off_w = layer == 0 ? kOffW3 : kOffW2, off_b = layer == 0 ? kOffB3 : kOffB2;
    if (g == 3) part[off_b + r] = tr_row_sum(sm.dzt, r);
    ok = tr_wait(sm, phase);  // (dzt and act are read; the next dZ may overwrite them)
    if (!ok) break;
    // dW (lane = output unit) into the tile's partial gradient
    float v[32];
    tmem_ld32(d_a + tlane + (uint32_t)col0, v);
    float *dst = part + off_w + col0 * kHid + r;  // [in][out] (param_of_partial)
#pragma unroll
    for (int i = 0; i < 32; ++i) dst[i * kHid] = v[i];
  }
  if (ok) {
    // ---- layer 1 (CUDA cores): dZ1 = dH1 * mask1 -> dzt; dW1[unit][c] = sum_row dZ1[row][unit] x[row][c], db1 ----
    {
      float v[32];
      tmem_ld32(d_b + tlane + (uint32_t)col0, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = (mask1 >> i) & 1u ? v[i] : 0.0f;
      tr_store32(nullptr, sm.dzt, r, col0, v);
    }
    __syncthreads();
    // group g: input g, or (g = 3) the bias
    float s = 0.0f;
    if (g < 3) {
#pragma unroll 4
      for (int c = 0; c < kTrainRows / 8; ++c) {
        const uint4 q = *reinterpret_cast<const uint4 *>(sm.dzt + tr_offset(r, 8 * c));
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q);
        const float4 *xp = reinterpret_cast<const float4 *>(sm.x[g] + 8 * c);
        const float4 xa = xp[0], xb = xp[1];
        const float xs[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(h[i]);
          s = fmaf(f.x, xs[2 * i], s);
          s = fmaf(f.y, xs[2 * i + 1], s);
        }
      }
    } else {
      s = tr_row_sum(sm.dzt, r);
    }
    part[g < 3 ? kOffW1 + 3 * r + g : kOffB1 + r] = s;
  }
  if (!ok && threadIdx.x == 0 && a.status) atomicOr(a.status, kStatusWaitTimeout);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(sm.tmem_base, kTrCols);
}

size_t mlp_train_smem_bytes() { return sizeof(TrainSmem); }

cudaError_t launch_mlp_train(const MlpTrainArgs &a, int n_tiles, bool overlap, cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_mlp_train, (int)sizeof(TrainSmem), configured);
  if (e != cudaSuccess) return e;
  return launch_overlapped(overlap, k_mlp_train, n_tiles, kTrThreads, sizeof(TrainSmem), st, a);
}

}  // namespace gg
