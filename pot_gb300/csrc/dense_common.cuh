// Shared pieces of the dense Sinkhorn kernels (dense.cu, fused.cuh).
#pragma once
#include "common.cuh"

namespace otg {

template <typename T> struct Pair { T mx, s; };

template <typename T>
__device__ __forceinline__ Pair<T> ldcg_pair(const Pair<T>* p) {
  const T* q = reinterpret_cast<const T*>(p);
  return Pair<T>{__ldcg(q), __ldcg(q + 1)};
}

// Per-thread maxima carried out of a pass (stabilised: d0; unbalanced:
// |u_new - u_old|, |u_new|, |u_old|).
struct Track {
  double d0 = -INFINITY, d1 = -INFINITY, d2 = -INFINITY;
};

// Order-preserving map of doubles to unsigned keys (atomicMax on keys = max
// on values; key 0 is below every value).
__device__ __forceinline__ unsigned long long order_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double key_value(unsigned long long k) {
  return (k >> 63) ? __longlong_as_double((long long)(k & 0x7fffffffffffffffull)) : __longlong_as_double((long long)~k);
}

// Block-wide max of one value per thread, then one atomicMax per CTA.  All
// threads of the block call it.
__device__ inline void block_max_atomic(double x, unsigned long long* slot) {
  __shared__ double red[32];
  x = warp_max(x);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = -INFINITY;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t = fmax(t, red[k]);
    if (t != -INFINITY) atomicMax(slot, order_key(t));
  }
  __syncthreads();
}

}  // namespace otg
