// host_warp.h - the CUDA built-ins of the device headers for a host compiler, as a warp of one lane.
//
// Included before the headers of opengate_gb300/csrc, it lets a test call their device functions on
// the CPU: a warp vote is the lane's own, an exchange gives its own value back, a barrier does nothing.
// (With no CUDA compiler the toolkit's headers define __device__ and the like as nothing.)
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#define __noinline__ __attribute__((noinline))

using std::max;
using std::min;

template <typename To, typename From>
inline To host_bits(From v) {
  static_assert(sizeof(To) == sizeof(From), "a reinterpretation");
  To t;
  std::memcpy(&t, &v, sizeof(t));
  return t;
}

struct HostIndex {
  unsigned x;
};
static const HostIndex threadIdx = {0u}, blockIdx = {0u}, gridDim = {1u}, blockDim = {1u};

inline unsigned __float_as_uint(float v) { return host_bits<unsigned>(v); }
inline float __uint_as_float(unsigned v) { return host_bits<float>(v); }
inline float __int_as_float(int v) { return host_bits<float>(v); }
inline long long __double_as_longlong(double v) { return host_bits<long long>(v); }
inline double __longlong_as_double(long long v) { return host_bits<double>(v); }
inline unsigned long long __float2ull_rn(float v) { return (unsigned long long)std::nearbyint(v); }
inline unsigned long long __double2ull_rn(double v) { return (unsigned long long)std::nearbyint(v); }
inline float __fsqrt_rn(float v) { return std::sqrt(v); }
inline double __dsqrt_rn(double v) { return std::sqrt(v); }
inline float __frcp_rn(float v) { return 1.0f / v; }
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
template <typename T>
inline T __ldg(const T *p) {
  return *p;
}

inline unsigned __ballot_sync(unsigned, int p) { return p ? 1u : 0u; }
inline int __any_sync(unsigned, int p) { return p != 0; }
template <typename T>
inline T __shfl_sync(unsigned, T v, int) {
  return v;
}
template <typename T>
inline T __shfl_up_sync(unsigned, T v, unsigned) {
  return v;
}
inline unsigned __reduce_add_sync(unsigned, unsigned v) { return v; }
inline void __syncwarp() {}
inline void __syncthreads() {}
template <typename T, typename U>
inline T atomicAdd(T *p, U v) {
  const T old = *p;
  *p = (T)(old + v);
  return old;
}
template <typename T, typename U>
inline T atomicOr(T *p, U v) {
  const T old = *p;
  *p = (T)(old | v);
  return old;
}
inline size_t __cvta_generic_to_shared(const void *) { return 0; }
