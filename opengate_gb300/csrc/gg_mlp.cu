// gg_mlp.cu - optimiser step and batch inference of the ARF network.
//
// One training step over a batch of B rows (B a multiple of kTrainRows):
//   k_mlp_train (gg_mlp_train.cu): one CTA per tile of 128 rows on the
//     5th-generation tensor cores - forward, softmax cross-entropy, backward;
//     each CTA writes its tile's parameter gradient (FP32, all kNParams) and
//     loss sum;
//   k_mlp_adam: one thread per parameter - the tile gradients summed in tile
//     order (deterministic), Adam update of the FP32 parameters, and the BF16
//     copies of W2 / W3 / W4 (row-major, tensor-core operands, transposed
//     operands) refreshed for the next step.
// Batch inference (k_mlp_predict) runs the forward pass on tcgen05 (gg_mlp_tc.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_internal.h"
#include "gg_mlp.cuh"
#include "gg_mlp_tc.cuh"

namespace gg {

// Sum of the tile gradients (tile order) and one Adam step; refreshes the BF16
// copies.  The last block adds the tiles' losses (tile order) instead.  Bound by
// the latency of the tile loads: 64 tiles, cold cache, 11.4 -> 8.4 us with 16 of
// them in flight per thread and the loss off the parameters' path.
constexpr int kAdamThreads = 128;
constexpr int kAdamBlocks = (kNParams + kAdamThreads - 1) / kAdamThreads;

__global__ void __launch_bounds__(kAdamThreads) k_mlp_adam(MlpAdamArgs a) {
  cudaTriggerProgrammaticLaunchCompletion();  // (the next step's kernel may set itself up)
  cudaGridDependencySynchronize();            // the tile gradients
  if (blockIdx.x == kAdamBlocks) {
    if (!a.loss_acc || threadIdx.x >= 32) return;
    double s = 0.0;
    for (int t0 = 0; t0 < a.n_tiles; t0 += 32) {
      const int t = t0 + (int)threadIdx.x, n = min(32, a.n_tiles - t0);
      const float l = t < a.n_tiles ? a.loss_part[t] : 0.0f;
      for (int k = 0; k < n; ++k) s += (double)__shfl_sync(0xffffffffu, l, k);
    }
    if (threadIdx.x == 0) *a.loss_acc += s;
    return;
  }
  const int q = blockIdx.x * kAdamThreads + threadIdx.x;  // in the tile gradients' order, as the moments
  if (q >= kNParams) return;
  const int p = param_of_partial(q);
  const bool update = a.lr != 0.0f;  // (else: gradient only)
  float m = 0.0f, v = 0.0f, w0 = 0.0f;
  if (update) {
    m = a.m[q];
    v = a.v[q];
    w0 = a.params[p];
  }
  float g = 0.0f;
  const float *part = a.partial + q;
  int t = 0;
  for (; t + 16 <= a.n_tiles; t += 16) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = part[(size_t)(t + i) * kNParams];
#pragma unroll
    for (int i = 0; i < 16; ++i) g += x[i];
  }
  for (; t < a.n_tiles; ++t) g += part[(size_t)t * kNParams];
  if (a.grad_out) a.grad_out[p] = g;
  if (!update) return;
  m = a.beta1 * m + (1.0f - a.beta1) * g;
  v = a.beta2 * v + (1.0f - a.beta2) * g * g;
  a.m[q] = m;
  a.v[q] = v;
  const float mh = m * a.c1, vh = v * a.c2;
  const float w = w0 - a.lr * mh / (sqrtf(vh) + a.eps);
  a.params[p] = w;
  bf16_store_weight(a.wbf, p, w);
}

// The first row (E, theta, phi, class) that is not finite or whose class is not
// a whole number in [0, n_classes): its number into *bad (atomicMin).
__global__ void __launch_bounds__(256) k_check_rows(const float4 *rows, uint64_t n, float n_classes,
                                                    unsigned long long *bad) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const float4 r = rows[i];
    const bool ok = isfinite(r.x) && isfinite(r.y) && isfinite(r.z) && r.w >= 0.0f && r.w < n_classes && r.w == floorf(r.w);
    if (!ok) atomicMin(bad, (unsigned long long)i);
  }
}

// BF16 copies of W2 / W3 / W4 from the FP32 parameters.
__global__ void k_mlp_to_bf16(const float *params, __nv_bfloat16 *wbf) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < kHid * kHid) {
    bf16_store_weight(wbf, kOffW2 + e, params[kOffW2 + e]);
    bf16_store_weight(wbf, kOffW3 + e, params[kOffW3 + e]);
  }
  if (e < kOutPad * kHid) bf16_store_weight(wbf, kOffW4 + e, params[kOffW4 + e]);
}

// Class probabilities of n rows on the 5th-generation tensor cores
// (gg_mlp_tc.cuh): each warpgroup of a CTA takes tiles of 128 rows in turn.
__global__ void __launch_bounds__(kTcThreads, 1)
    k_mlp_predict(MlpTrainArgs a, float *out, uint64_t n, unsigned int *status) {
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  TcNetSmem &sm = *reinterpret_cast<TcNetSmem *>(tc_smem_raw);
  const bool ready = tc_net_prepare(sm, a.params, a.wbf);
  const int g = threadIdx.x >> 7, r = threadIdx.x & 127;
  uint32_t phase = 0;
  const uint64_t n_tiles = (n + kTcRows - 1) / kTcRows;
  if (!ready && threadIdx.x == 0) atomicOr(status, kStatusWaitTimeout);
  for (uint64_t t = (uint64_t)blockIdx.x * kTcGroups + g; ready && t < n_tiles;
       t += (uint64_t)gridDim.x * kTcGroups) {
    const uint64_t row = t * kTcRows + r;
    const float4 v = row < n ? a.rows[row] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float x0 = (v.y - a.mean[0]) * a.inv_std[0];
    const float x1 = (v.z - a.mean[1]) * a.inv_std[1];
    const float x2 = (v.x - a.mean[2]) * a.inv_std[2];
    float p[16];
    if (!tc_net_forward(sm, g, r, phase, x0, x1, x2, p)) {
      if (r == 0) atomicOr(status, kStatusWaitTimeout);
      break;
    }
    tc_softmax(p, a.n_classes);
    if (row < n) {
#pragma unroll
      for (int c = 0; c < 16; ++c)
        if (c < a.n_classes) out[row * a.n_classes + c] = p[c];
    }
  }
  tc_net_teardown(sm);
}

cudaError_t launch_mlp_adam(const MlpAdamArgs &a, bool overlap, cudaStream_t st) {
  return launch_overlapped(overlap, k_mlp_adam, kAdamBlocks + 1, kAdamThreads, 0, st, a);
}

cudaError_t launch_check_rows(const float4 *rows, uint64_t n, int n_classes, unsigned long long *bad, int n_sm,
                              cudaStream_t st) {
  k_check_rows<<<n_sm * 4, 256, 0, st>>>(rows, n, (float)n_classes, bad);
  return cudaGetLastError();
}

cudaError_t launch_mlp_to_bf16(const float *params, __nv_bfloat16 *wbf, cudaStream_t st) {
  k_mlp_to_bf16<<<(kHid * kHid + 255) / 256, 256, 0, st>>>(params, wbf);
  return cudaGetLastError();
}

size_t mlp_tc_smem_bytes() { return sizeof(TcNetSmem); }

cudaError_t launch_mlp_predict(const MlpTrainArgs &a, float *out, uint64_t n, int grid, unsigned int *status,
                               cudaStream_t st) {
  static unsigned long long configured = 0;
  cudaError_t e = configure_smem(k_mlp_predict, (int)sizeof(TcNetSmem), configured);
  if (e != cudaSuccess) return e;
  k_mlp_predict<<<grid, kTcThreads, sizeof(TcNetSmem), st>>>(a, out, n, status);
  return cudaGetLastError();
}

}  // namespace gg
