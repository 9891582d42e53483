// Building blocks of the kernels that read the cost once per iteration
// (fused_impl.cuh, multi_fused.cuh): 16-byte vectors in registers, reductions
// of several rows at once, ring copies, a bounded grid barrier.
#pragma once
#include "dense_common.cuh"
#include "tma.cuh"

namespace otg {

constexpr int FU_THREADS = 256, FU_WARPS = 8;
// Rows of a batch for NK vectors per row and thread: up to 16 vectors (256
// bytes) of entries in a thread's registers.
__host__ __device__ constexpr int fu_rb(int nk) { return nk > 8 ? 1 : nk > 4 ? 2 : nk > 2 ? 4 : 8; }

struct FuRow {                 // this thread's place
  int r0, r1;                  // rows of the CTA
  int ga, gb;                  // rows of its group
  int live;                    // groups with rows
  int g, NG, gt, tg, warp, lane;
};

template <typename T>
__device__ __forceinline__ void fu_get(const T* p, T (&x)[Vec<T>::N]) {
  unpack(*reinterpret_cast<const typename Vec<T>::type*>(p), x);
}
__device__ __forceinline__ void fu_put(float* p, const float (&x)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ void fu_put(double* p, const double (&x)[2]) {
  *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
}

// A 16-byte vector in registers: two packed pairs of floats (the packed
// fp32x2 operations round each lane as the scalar ones), or two doubles.
template <typename T> struct FuV;
template <> struct FuV<float> {
  uint64_t a, b;
  struct S { uint64_t v; };  // a scalar for both lanes
  static __device__ __forceinline__ S all(float x) { return S{pack2(x, x)}; }
  static __device__ __forceinline__ FuV zero() { return FuV{0ull, 0ull}; }
  static __device__ __forceinline__ FuV lds(uint32_t p) {
    FuV r;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "r"(p) : "memory");
    return r;
  }
  // zeros where `on` is false
  static __device__ __forceinline__ FuV lds_if(uint32_t p, bool on) {
    FuV r;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.b64 %0, 0;\n\tmov.b64 %1, 0;\n\t"
        "@q ld.shared.v2.b64 {%0, %1}, [%2];\n\t}"
        : "=&l"(r.a), "=&l"(r.b) : "r"(p), "r"((int)on) : "memory");
    return r;
  }
  static __device__ __forceinline__ uint64_t ex(uint64_t t) {
    float lo, hi;
    unpack2(t, lo, hi);
    return pack2(ex2(lo), ex2(hi));
  }
  // this += x * r
  __device__ __forceinline__ void fma_s(const FuV& x, S r) { a = fma2(x.a, r.v, a); b = fma2(x.b, r.v, b); }
  // this += x * y
  __device__ __forceinline__ void fma_v(const FuV& x, const FuV& y) { a = fma2(x.a, y.a, a); b = fma2(x.b, y.b, b); }
  __device__ __forceinline__ void add_v(const FuV& x) { a = add2(a, x.a); b = add2(b, x.b); }
  // exp2(x c + v + h)
  static __device__ __forceinline__ FuV expo(const FuV& x, S c, const FuV& v, S h) {
    return FuV{ex(add2(fma2(x.a, c.v, v.a), h.v)), ex(add2(fma2(x.b, c.v, v.b), h.v))};
  }
  // exp2(x c)
  static __device__ __forceinline__ FuV gibbs(const FuV& x, S c) { return FuV{ex(mul2(x.a, c.v)), ex(mul2(x.b, c.v))}; }
  static __device__ __forceinline__ FuV arg(const FuV& x, S c, const FuV& v) { return FuV{fma2(x.a, c.v, v.a), fma2(x.b, c.v, v.b)}; }
  static __device__ __forceinline__ FuV ex_minus(const FuV& t, float m) {
    const uint64_t k = pack2(-m, -m);
    return FuV{ex(add2(t.a, k)), ex(add2(t.b, k))};
  }
  __device__ __forceinline__ void get(float (&x)[4]) const { unpack2(a, x[0], x[1]); unpack2(b, x[2], x[3]); }
  static __device__ __forceinline__ FuV of(const float (&x)[4]) { return FuV{pack2(x[0], x[1]), pack2(x[2], x[3])}; }
  __device__ __forceinline__ float sum() const { float x[4]; get(x); return (x[0] + x[1]) + (x[2] + x[3]); }
  __device__ __forceinline__ float max_with(float m) const { float x[4]; get(x); return fmaxf(fmax3(m, x[0], x[1]), fmaxf(x[2], x[3])); }
};
template <> struct FuV<double> {
  double a, b;
  struct S { double v; };
  static __device__ __forceinline__ S all(double x) { return S{x}; }
  static __device__ __forceinline__ FuV zero() { return FuV{0.0, 0.0}; }
  static __device__ __forceinline__ FuV lds(uint32_t p) {
    FuV r;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.a), "=d"(r.b) : "r"(p) : "memory");
    return r;
  }
  static __device__ __forceinline__ FuV lds_if(uint32_t p, bool on) {
    FuV r;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
        "mov.f64 %1, 0d0000000000000000;\n\t@q ld.shared.v2.f64 {%0, %1}, [%2];\n\t}"
        : "=&d"(r.a), "=&d"(r.b) : "r"(p), "r"((int)on) : "memory");
    return r;
  }
  __device__ __forceinline__ void fma_s(const FuV& x, S r) { a = fma(x.a, r.v, a); b = fma(x.b, r.v, b); }
  __device__ __forceinline__ void fma_v(const FuV& x, const FuV& y) { a = fma(x.a, y.a, a); b = fma(x.b, y.b, b); }
  __device__ __forceinline__ void add_v(const FuV& x) { a += x.a; b += x.b; }
  static __device__ __forceinline__ FuV expo(const FuV& x, S c, const FuV& v, S h) {
    return FuV{ex2(fma(x.a, c.v, v.a) + h.v), ex2(fma(x.b, c.v, v.b) + h.v)};
  }
  static __device__ __forceinline__ FuV gibbs(const FuV& x, S c) { return FuV{ex2(x.a * c.v), ex2(x.b * c.v)}; }
  static __device__ __forceinline__ FuV arg(const FuV& x, S c, const FuV& v) { return FuV{fma(x.a, c.v, v.a), fma(x.b, c.v, v.b)}; }
  static __device__ __forceinline__ FuV ex_minus(const FuV& t, double m) { return FuV{ex2(t.a - m), ex2(t.b - m)}; }
  __device__ __forceinline__ void get(double (&x)[2]) const { x[0] = a; x[1] = b; }
  static __device__ __forceinline__ FuV of(const double (&x)[2]) { return FuV{x[0], x[1]}; }
  __device__ __forceinline__ double sum() const { return a + b; }
  __device__ __forceinline__ double max_with(double m) const { return fmax(m, fmax(a, b)); }
};

// Ring of the streamed form.  Chunk j of a group's pass is half (j & 1) of its
// row j / 2, `half` elements per slot.  The chunks of the next pass follow
// those of this one (the cost does not change), so the ring never runs dry
// over the hand-over.  Chunk j into `slot`; `rows`: rows of the group, M0: its
// first one.
template <typename T>
__device__ __forceinline__ void fu_issue(const T* M0, int64_t ldm, int mv, int half, int rows, T* slots, uint64_t* full, int j,
                                         int slot) {
  const int nch = 2 * rows;
  while (j >= nch) j -= nch;
  const int c0 = (j & 1) * half, cols = min(half, mv - c0);
  if (cols > 0) {
    mbar_arrive_expect_tx(full + slot, (uint32_t)(cols * (int)sizeof(T)));
    bulk_g2s(slots + slot * half, M0 + (int64_t)(j >> 1) * ldm + c0, (uint32_t)(cols * (int)sizeof(T)), full + slot);
  } else {
    mbar_arrive(full + slot);
  }
}

// ---------------------------------------------------------------------------
// Reductions over RB rows at once.  Each lane brings its share of every row;
// after log2(RB) halving steps and the rest of the butterfly, lane l holds
// the warp's value of row l / LPR.
// ---------------------------------------------------------------------------
template <typename T, bool MAX> __device__ __forceinline__ T fu_op(T a, T b) { return MAX ? fmax(a, b) : a + b; }

template <typename T, int RB, bool MAX>
__device__ __forceinline__ T fu_scatter(T (&s)[RB], int lane) {
  int o = 16;
#pragma unroll
  for (int h = RB / 2; h >= 1; h /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const T keep = up ? s[i + h] : s[i], give = up ? s[i] : s[i + h];
      s[i] = fu_op<T, MAX>(keep, __shfl_xor_sync(0xffffffffu, give, o));
    }
    o >>= 1;
  }
  T x = s[0];
#pragma unroll
  for (int q = 16 / RB; q > 0; q >>= 1) x = fu_op<T, MAX>(x, __shfl_xor_sync(0xffffffffu, x, q));
  return x;
}

// ... over the G warps of the group: lane l of every warp gets the group's
// value of row l / LPR.  The scratch alternates, one barrier per call.
template <typename T, int RB, bool MAX, int RS>
__device__ __forceinline__ T fu_group(T (&s)[RB], const FuRow& R, int G, T (*red)[FU_WARPS][RS], int& par) {
  constexpr int LPR = 32 / RB;
  T x = fu_scatter<T, RB, MAX>(s, R.lane);
  if (G == 1) return x;
  const int row = R.lane / LPR, l = R.lane % LPR, w0 = R.g * G;
  if (l == 0) red[par][R.warp][row] = x;
  named_bar(1 + R.g, R.gt);
  T t = MAX ? T(-INFINITY) : T(0);
  for (int q = l; q < G; q += LPR) t = fu_op<T, MAX>(t, red[par][w0 + q][row]);
#pragma unroll
  for (int q = LPR / 2; q > 0; q >>= 1) t = fu_op<T, MAX>(t, __shfl_xor_sync(0xffffffffu, t, q));
  par ^= 1;
  return t;
}

// x >= lim > 0; false for a NaN.  (Doubles by integers: an FP64 comparison
// issues at two lanes per clock.)
__device__ __forceinline__ bool fu_at_least(float x, float lim) { return x >= lim; }
__device__ __forceinline__ bool fu_at_least(double x, double lim) {
  const long long b = __double_as_longlong(x);
  return b >= __double_as_longlong(lim) && b <= 0x7ff0000000000000ll;
}
// 2^k, a normal number.
template <typename T> __device__ __forceinline__ T exp2_of(int k);
template <> __device__ __forceinline__ float exp2_of<float>(int k) { return __int_as_float((127 + k) << 23); }
template <> __device__ __forceinline__ double exp2_of<double>(int k) { return __hiloint2double((1023 + k) << 20, 0); }

template <typename T>
__device__ __forceinline__ bool fu_near_one(T t) { return t >= T(9.313225746154785e-10) && t <= T(1073741824.0); }  // 2^-30, 2^30

// Grid barrier with one counter that
// only grows (the launch's control block starts at zero).  Bounded.
__device__ __forceinline__ bool fu_barrier(unsigned* bar, unsigned& gen, int* abort_flag, uint64_t timeout_ns) {
  __shared__ int s_ok;
  __syncthreads();
  gen += gridDim.x;
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    atomicAdd(bar, 1u);
    if ((int)(ld_acquire(bar) - gen) < 0) {
      const uint64_t t0 = globaltimer();
      unsigned spins = 0;
      while ((int)(ld_acquire(bar) - gen) < 0) {
        if ((++spins & 255u) == 0) {
          if (ld_acquire_i(abort_flag)) { ok = 0; break; }
          if (globaltimer() - t0 > timeout_ns) { atomicExch(abort_flag, 1); ok = 0; break; }
        }
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

}  // namespace otg
