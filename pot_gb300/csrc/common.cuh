// Shared device helpers for the entropic-OT kernels (sm_103a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include "exp2_table.cuh"
#include "log2_table.cuh"

#define OTG_LOG2E 1.4426950408889634
#define OTG_LN2 0.6931471805599453

namespace otg {

// ---------------------------------------------------------------------------
// exp2 / log2 in the working precision.  fp32 uses the MUFU ex2 instruction
// (PTX ex2.approx.ftz.f32, relative error about 2^-22).
//
// fp64: FP64 issues at two lanes per clock and SM here, so what an
// exponential costs is its number of FP64 operations.  Table-driven form (P.
// T. P. Tang, ACM TOMS 15 (1989) 144-157): x = n + j / 128 + f, |f| <= 1 /
// 256, 2^x = 2^n (T_j + (T_j p(f) + t_j)) with T_j + t_j = 2^(j/128) to 106
// bits and p the series of 2^f - 1 to degree 5 (the next term is 6e-19): ten
// FP64 operations, error below 0.52 ulp.  The table is read through L1.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^(k / 128 + f), the result in the normal range.
__device__ __forceinline__ double exp2_core(int k, double f) {
  const double2 T = __ldg(EXP2_TABLE + (k & 127));
  double p = fma(f, 0x1.5d87fe78a6731p-10, 0x1.3b2ab6fba4e77p-7);
  p = fma(f, p, 0x1.c6b08d704a0c0p-5);
  p = fma(f, p, 0x1.ebfbdff82c58fp-3);
  p = fma(f, p, 0x1.62e42fefa39efp-1);
  p *= f;
  const double r = T.x + fma(T.x, p, T.y);
  return __hiloint2double(__double2hiint(r) + (k >> 7) * (1 << 20), __double2loint(r));
}
__device__ __forceinline__ double ex2(double x) {
  const int hx = __double2hiint(x);
  const unsigned ah = (unsigned)hx & 0x7fffffffu;
  double y = x, back = 0.0;
  if (ah >= 0x408ff000u) {  // |x| >= 1022: the exponent in two steps
    if (ah >= 0x40913000u) {  // |x| >= 1100, infinities, NaN
      if (ah > 0x7ff00000u || (ah == 0x7ff00000u && __double2loint(x) != 0)) return x + x;
      return hx < 0 ? 0.0 : __hiloint2double(0x7ff00000, 0);
    }
    y = hx < 0 ? x + 128.0 : x - 128.0;
    back = hx < 0 ? 0x1p-128 : 0x1p128;
  }
  const double t = y + 0x1.8p45;  // multiples of 1 / 128
  const double s = exp2_core(__double2loint(t), y - (t - 0x1.8p45));
  return back == 0.0 ? s : s * back;
}

// x^y for 0 < y <= 1 (anything else: the library's).  A chain of some 40 FP64
// operations (500 x 700 unbalanced in float64: 27.1 -> 26.4 us per iteration): a
// table-driven logarithm (P. T. P. Tang, ACM TOMS 16 (1990) 378-400) with the
// leading terms in two parts, then the exponential above.  Within 0.52 ulp.
__device__ __forceinline__ float pow_unit(float x, float y) { return pow(x, y); }
__device__ __forceinline__ double pow_unit(double x, double y) {
  const int hx = __double2hiint(x), hy = __double2hiint(y);
  if ((unsigned)(hx - 0x00100000) >= 0x7fe00000u || hy < 0x3c000000 || !(y <= 1.0)) return pow(x, y);
  const int t = hx - 0x3fe6a09e, e = t >> 20;
  const double m = __hiloint2double(hx - e * (1 << 20), __double2loint(x));
  const int i = __double2loint(m + 0x1.8p45) - 90;
  const double2 T = __ldg(LOG2_TABLE + i);
  const double r = fma(m, T.x, -1.0);
  // log2(1 + r): the linear term in two parts, the others to r^8
  const double h = r * 0x1.71547652b82fep+0, l = fma(r, 0x1.777d0ffda0d24p-56, fma(r, 0x1.71547652b82fep+0, -h));
  const double r2 = r * r;
  const double a = fma(r, 0x1.ec709dc3a03fdp-2, -0x1.71547652b82fep-1), b = fma(r, 0x1.2776c50ef9bfep-2, -0x1.71547652b82fep-2), c = fma(r, 0x1.a61762a7aded9p-3, -0x1.ec709dc3a03fdp-3);
  const double q = r2 * fma(r2, fma(r2, fma(r2, -0x1.71547652b82fep-3, c), b), a);
  // (e as a double by its bits: a conversion costs four FP64 operations)
  const double A = (__hiloint2double(0x43300000, e ^ (int)0x80000000u) - 0x1.000008p52) + T.y, s = A + h;
  const double lo = ((A - s) + h) + (l + (__ldg(LOG2_REST + i) + q));
  const double z = y * s, zl = fma(y, lo, fma(y, s, -z));
  const double u = z + 0x1.8p45;
  return exp2_core(__double2loint(u), (z - (u - 0x1.8p45)) + zl);
}
__device__ __forceinline__ float lg2(float x) { return log2f(x); }
__device__ __forceinline__ double lg2(double x) { return log2(x); }

// Packed fp32x2 arithmetic (sm_100 family): one instruction for a pair of
// floats in a 64-bit register, each lane rounded as the scalar operation.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// max of three floats in one instruction (NaN inputs handled as by fmaxf)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// float -> double by integer operations (exact; denormals, infinities and NaN
// by the conversion): the conversion issues at half a lane per clock and SM
// here, a quarter of the rate of FP64 arithmetic.
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), e = b & 0x7f800000u, s = b & 0x80000000u;
  if ((b << 1) == 0u) return __hiloint2double((int)s, 0);
  if (e == 0u || e == 0x7f800000u) return (double)x;
  return __hiloint2double((int)(s | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ double widen(double x) { return x; }

// Running sums that lose nothing next to float64 ones.  float: two lanes of
// packed fp32 operations (even and odd terms), each with the rounding errors of
// its additions in a second float (D. E. Knuth, TAOCP 2, 4.2.2): seven packed
// operations for two terms, where widening and an FP64 addition issue at two
// lanes per clock and SM; double: a plain sum.
template <typename T> struct Sum2;
template <> struct Sum2<float> {
  uint64_t hi = 0ull, lo = 0ull;
  __device__ __forceinline__ void add_(uint64_t x) {
    const uint64_t m1 = pack2(-1.f, -1.f), s = add2(hi, x), b = fma2(hi, m1, s);
    lo = add2(lo, add2(fma2(fma2(b, m1, s), m1, hi), fma2(b, m1, x)));
    hi = s;
  }
  __device__ __forceinline__ void add(float x, float y) { add_(pack2(x, y)); }
  // + x0 y0, x1 y1, the products' roundings kept too
  __device__ __forceinline__ void fma_(float x0, float y0, float x1, float y1) {
    const uint64_t x = pack2(x0, x1), y = pack2(y0, y1), p = mul2(x, y);
    lo = add2(lo, fma2(x, y, fma2(p, pack2(-1.f, -1.f), 0ull)));
    add_(p);
  }
  // (an infinite sum has no error term)
  __device__ __forceinline__ double value() const {
    float h0, h1, l0, l1;
    unpack2(hi, h0, h1);
    unpack2(lo, l0, l1);
    const double h = widen(h0) + widen(h1);
    return isfinite(h0) && isfinite(h1) ? h + widen(l0 + l1) : h;
  }
};
template <> struct Sum2<double> {
  double hi = 0.0;
  __device__ __forceinline__ void add(double x, double y) { hi += x; hi += y; }
  __device__ __forceinline__ void fma_(double x0, double y0, double x1, double y1) { hi = fma(x1, y1, fma(x0, y0, hi)); }
  __device__ __forceinline__ double value() const { return hi; }
};

template <typename T> struct Vec;
template <> struct Vec<float> { using type = float4; static constexpr int N = 4; };
template <> struct Vec<double> { using type = double2; static constexpr int N = 2; };

__device__ __forceinline__ void unpack(const float4& q, float* o) { o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w; }
__device__ __forceinline__ void unpack(const double2& q, double* o) { o[0] = q.x; o[1] = q.y; }

// Streaming 128-bit load that does not allocate in L1 (the cost matrix is
// read once per pass).
__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ double2 ld_stream(const double2* p) {
  double2 r;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0,%1}, [%2];"
               : "=d"(r.x), "=d"(r.y) : "l"(p));
  return r;
}

// ---------------------------------------------------------------------------
// (max, sum) pairs of a base-2 log-sum-exp: the value is  mx + log2(s).
// An empty pair is (-inf, 0).  Merging is associative and commutative, so
// partial pairs from any split of a row or column combine in any order.
// ---------------------------------------------------------------------------
// A NaN maximum is dropped by fmax but poisons the sum through ex2(NaN), so
// NaN inputs still give a NaN result, as they do in the reference.
template <typename T>
__device__ __forceinline__ void lse_merge(T& mx, T& s, T mx2, T s2) {
  T nm = fmax(mx, mx2);
  if (nm == -INFINITY) return;  // both empty
  s = s * ex2(mx - nm) + s2 * ex2(mx2 - nm);
  mx = nm;
}

template <typename T>
__device__ __forceinline__ T lse_value(T mx, T s) {
  if (mx == -INFINITY) return -INFINITY;
  return mx + lg2(s);
}

// Merge `cnt` (max, sum) pairs stored as consecutive (mx, s) values at
// p, p + stride, p + 2 stride, ...  (L2-coherent loads, eight independent
// loads in flight before the dependent merges).
template <typename T>
__device__ __forceinline__ void lse_merge_strided(T& mx, T& s, const T* p, int64_t stride, int cnt) {
  int r = 0;
  for (; r + 8 <= cnt; r += 8) {
    T m8[8], s8[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { m8[k] = __ldcg(p + (r + k) * stride); s8[k] = __ldcg(p + (r + k) * stride + 1); }
#pragma unroll
    for (int k = 0; k < 8; ++k) lse_merge(mx, s, m8[k], s8[k]);
  }
  for (; r < cnt; ++r) lse_merge(mx, s, __ldcg(p + r * stride), __ldcg(p + r * stride + 1));
}

template <typename T>
__device__ __forceinline__ T sum_strided(const T* p, int64_t stride, int cnt) {
  T acc = 0;
  int r = 0;
  for (; r + 8 <= cnt; r += 8) {
    T v8[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v8[k] = __ldcg(p + (r + k) * stride + 1);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += v8[k];
  }
  for (; r < cnt; ++r) acc += __ldcg(p + r * stride + 1);
  return acc;
}

template <typename T>
__device__ __forceinline__ void warp_lse(T& mx, T& s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    T m2 = __shfl_xor_sync(0xffffffffu, mx, o);
    T s2 = __shfl_xor_sync(0xffffffffu, s, o);
    lse_merge(mx, s, m2, s2);
  }
}

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <typename T>
__device__ __forceinline__ T warp_max(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Maximum of a (never NaN) and b, both non-negative or -inf, a NaN b dropped
// as by fmax.  Doubles by integer comparison: FP64 comparisons are FP64
// operations, two lanes per clock (the unbalanced stop test in float64: 100 x
// 100 21.7 -> 15.0 us per iteration, 500 x 700 26.4 -> 18.6).
__device__ __forceinline__ float pos_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double pos_max(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  return y > x && y <= 0x7ff0000000000000ll ? b : a;
}
template <typename T>
__device__ __forceinline__ T warp_pos_max(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = pos_max(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

__device__ __forceinline__ int warp_or(int x) { return __any_sync(0xffffffffu, x) ? 1 : 0; }

// ---------------------------------------------------------------------------
// Reductions in a fixed order.  Floating-point addition is not associative,
// so a sum whose terms arrive through atomics changes from run to run in its
// last bits; a stopping test on such a sum can then stop at a different
// iteration.  Every error that feeds a stop decision is therefore summed in
// an order fixed by the data layout alone: partials are stored in fixed
// slots and summed by these helpers.
//
// warp_sum's xor butterfly combines partner values commutatively at every
// step, so all lanes hold the same, order-fixed value.
// ---------------------------------------------------------------------------
// Block sum of one double per thread; every thread gets the result.  All
// threads of the block call it.
__device__ __forceinline__ double block_sum_fixed(double x) {
  __shared__ double red[33];
  x = warp_sum(x);
  __syncthreads();  // red may still be read by a previous call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// Sum of p[0 .. cnt) by one block (thread t folds t, t + blockDim, ... in
// increasing order); every thread gets the result.
__device__ __forceinline__ double block_sum_slots(const double* p, int64_t cnt) {
  double x = 0.0;
  for (int64_t i = threadIdx.x; i < cnt; i += blockDim.x) x += __ldcg(p + i);
  return block_sum_fixed(x);
}

// *out = sum of slots[0 .. cnt) in a fixed order; launch with ONE block of
// BS threads.  (A template, so that every translation unit may include it.)
template <int BS>
__global__ void __launch_bounds__(BS) slot_sum_kernel(const double* __restrict__ slots, int64_t cnt, double* out) {
  const double t = block_sum_slots(slots, cnt);
  if (threadIdx.x == 0) *out = t;
}

// ---------------------------------------------------------------------------
// Bounded grid barrier for cooperative (co-resident) launches.
// bar[0] counts arrivals, bar[1] is the generation.  A block that waits
// longer than `timeout_ns` (globaltimer) sets *abort and leaves; callers check
// *abort after every barrier and return, so no wait is unbounded.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_acquire_i(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned nblocks, int* abort_flag,
                                             uint64_t timeout_ns) {
  __syncthreads();
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned gen = ld_acquire(bar + 1);
    __threadfence();
    unsigned arrived = atomicAdd(bar, 1u);
    if (arrived == nblocks - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      uint64_t t0 = globaltimer();
      unsigned spins = 0;
      while (ld_acquire(bar + 1) == gen) {
        if (++spins > 64) __nanosleep(64);
        if ((spins & 255u) == 0) {
          if (ld_acquire_i(abort_flag)) { ok = 0; break; }
          if (globaltimer() - t0 > timeout_ns) { atomicExch(abort_flag, 1); ok = 0; break; }
        }
      }
    }
    __threadfence();
    if (ld_acquire_i(abort_flag)) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

}  // namespace otg
