// gg_mlp.cuh - the ARF network: parameter layout and BF16 weight copies.
//
// Network (restating the garf ARF model used by the reference's ARFActor,
// opengate/actors/arfactors.py:349-415): input x = (theta deg, phi deg, E MeV)
// standardised with the training-set mean / std, three hidden layers of 128
// ReLU units, a linear output of n_classes logits (class 0 = no energy
// window, class k = window k) and a softmax.
//
// Parameters are one FP32 array (offsets below).  Layers 2-4 run on the
// 5th-generation tensor cores (gg_mlp_tc.cuh, gg_mlp_train.cu) from BF16
// copies of their weights with FP32 accumulation; layer 1 (3 inputs) runs on
// the CUDA cores in FP32.  Activations between layers are stored as BF16.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace gg {

constexpr int kHid = 128;     // hidden units
constexpr int kOutPad = 16;   // output logits padded to one n16 tile pair

// FP32 parameter layout
constexpr int kOffW1 = 0;                        // [128][3]
constexpr int kOffB1 = kOffW1 + kHid * 3;        // [128]
constexpr int kOffW2 = kOffB1 + kHid;            // [128][128] (out, in)
constexpr int kOffB2 = kOffW2 + kHid * kHid;     // [128]
constexpr int kOffW3 = kOffB2 + kHid;            // [128][128]
constexpr int kOffB3 = kOffW3 + kHid * kHid;     // [128]
constexpr int kOffW4 = kOffB3 + kHid;            // [16][128] (rows >= n_classes stay 0)
constexpr int kOffB4 = kOffW4 + kOutPad * kHid;  // [16]
constexpr int kNParams = kOffB4 + kOutPad;       // 35600

// Tile gradients (MlpTrainArgs::partial) and Adam moments keep W2 and W3 as [in]
// [out]: thread `out` of the training kernel reads one row of dW from tensor
// memory, and its stores of one column are contiguous over the lanes.  The
// parameter of entry q:
__host__ __device__ constexpr int param_of_partial(int q) {
  const int off = q >= kOffW2 && q < kOffB2 ? kOffW2 : (q >= kOffW3 && q < kOffB3 ? kOffW3 : -1);
  if (off < 0) return q;
  const int i = (q - off) / kHid, o = (q - off) % kHid;
  return off + o * kHid + i;
}

// BF16 weight copies used by the tensor cores: W2, W3, W4 back to back as
// 5th-generation tensor-core operands (K-major core matrices, gg_tc.cuh), so
// that one bulk copy per matrix stages them in shared memory
constexpr int kBfW2 = 0;
constexpr int kBfW3 = kHid * kHid;
constexpr int kBfW4 = 2 * kHid * kHid;
constexpr int kNBf = 2 * kHid * kHid + kOutPad * kHid;
// ... and transposed, W^T[in][out] (K = out; W4^T is 128 x 16), the B operands
// of the backward pass dH = dZ W, starting at element kTcTBf
constexpr int kTcTBf = kNBf;
constexpr int kNBfAll = 2 * kNBf;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Element offset of (n, k) in a K-major core-matrix operand with kk columns:
// the byte offset of the layout (gg_tc.cuh) / 2.
__host__ __device__ constexpr int tc_elem_k(int n, int k, int kk) {
  return (n >> 3) * (kk / 8) * 64 + (k >> 3) * 64 + (n & 7) * 8 + (k & 7);
}
__host__ __device__ constexpr int tc_elem(int n, int k) { return tc_elem_k(n, k, kHid); }

// Stores parameter p (a weight of W2, W3 or W4, value w) as BF16 in both copies.
__device__ __forceinline__ void bf16_store_weight(__nv_bfloat16 *wbf, int p, float w) {
  const __nv_bfloat16 b = __float2bfloat16_rn(w);
  int base, q;
  if (p >= kOffW2 && p < kOffB2) base = kBfW2, q = p - kOffW2;
  else if (p >= kOffW3 && p < kOffB3) base = kBfW3, q = p - kOffW3;
  else if (p >= kOffW4 && p < kOffB4) base = kBfW4, q = p - kOffW4;
  else return;
  const int o = q / kHid, i = q % kHid;
  wbf[base + tc_elem(o, i)] = b;
  // transposed: W^T[i][o], K = out units (128, or 16 for W4)
  const int kk = base == kBfW4 ? kOutPad : kHid;
  wbf[kTcTBf + base + tc_elem_k(i, o, kk)] = b;
}

}  // namespace gg
