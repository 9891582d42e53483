// What sinkhorn_knopp_unbalanced returns beside the plan, behind the solve:
// the vectors of its log and the total cost with its KL marginal penalties
// (ot/unbalanced/_sinkhorn.py:420-445).  As elementwise and reduction
// launches over the marginals this was 30 launches, 0.3 ms of a 2000 x 3000
// call; here four.
#include <algorithm>
#include "common.cuh"
#include "../../include/pot_gb300.h"

namespace otg {

// ut = alw u, vt = bew v (no weights: copies), lu = log(u + 1e-300), lv.
template <typename T>
__global__ void __launch_bounds__(256) unb_vectors_kernel(int64_t n, int64_t m, const T* u, const T* v, const T* alw, const T* bew,
                                                          T* ut, T* vt, T* lu, T* lv) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const T tiny = (T)(sizeof(T) == 8 ? 1e-300 : 0.0);  // (zero in float)
  if (i < n) {
    ut[i] = alw ? alw[i] * u[i] : u[i];
    lu[i] = log(u[i] + tiny);
  } else if (i < n + m) {
    const int64_t j = i - n;
    vt[j] = bew ? bew[j] * v[j] : v[j];
    lv[j] = log(v[j] + tiny);
  }
}

// Marginals of the plan: blocks below `rblocks` a warp per row (its KL term
// into krow), the others 128 columns of a range of rows (fp64 partial sums
// into cpart[range][m]).  Bound by two reads of the plan from L2; sums of
// eight entries with their rounding errors (Sum2), fp64 beyond.  2000 x 3000
// float32: 46 us for all of otg_unbalanced_total, 85 with every entry widened,
// 29 with float sums of eight entries.
constexpr int UB_SPLIT = 8;
template <typename T>
__global__ void __launch_bounds__(256) unb_marginals_kernel(const T* P, int64_t n, int64_t m, int64_t ldp, const T* a, int rows_on,
                                                            int64_t rblocks, double* krow, double* cpart) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x < rblocks) {
    const int64_t row = (int64_t)blockIdx.x * 8 + warp;
    if (row >= n || !rows_on) return;
    const T* p = P + row * ldp;
    double s = 0.0;
    for (int64_t j = lane; j < m; j += 256) {
      T x[8];
      Sum2<T> t;
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = j + 32 * k < m ? __ldg(p + j + 32 * k) : T(0);
#pragma unroll
      for (int k = 0; k < 8; k += 2) t.add(x[k], x[k + 1]);
      s += t.value();
    }
    s = warp_sum(s);
    if (lane == 0) krow[row] = s * log(s / (double)a[row] + 1e-16);
    return;
  }
  __shared__ double part[8][128];
  const int64_t b = blockIdx.x - rblocks, chunks = (m + 127) / 128;
  const int64_t c0 = (b % chunks) * 128, range = b / chunks;
  const int64_t r0 = n * range / UB_SPLIT, r1 = n * (range + 1) / UB_SPLIT;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t i = r0 + warp; i < r1; i += 64) {
    T x[8][4];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        x[k][q] = i + 8 * k < r1 && c0 + 32 * q + lane < m ? __ldg(P + (i + 8 * k) * ldp + c0 + 32 * q + lane) : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      Sum2<T> t;
#pragma unroll
      for (int k = 0; k < 8; k += 2) t.add(x[k][q], x[k + 1][q]);
      acc[q] += t.value();
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) part[warp][32 * q + lane] = acc[q];
  __syncthreads();
  if (threadIdx.x < 128 && c0 + threadIdx.x < m) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += part[w][threadIdx.x];
    cpart[range * m + c0 + threadIdx.x] = t;
  }
}

// Column KL terms, a block's sums of both sides into its slot.
template <typename T>
__global__ void __launch_bounds__(128) unb_terms_kernel(int64_t n, int64_t m, const T* b, int rows_on, int cols_on, const double* krow,
                                                        const double* cpart, double* slots) {
  const int64_t j = (int64_t)blockIdx.x * 128 + threadIdx.x;
  double c = 0.0, r = 0.0;
  if (cols_on && j < m) {
    double s = 0.0;
    for (int k = 0; k < UB_SPLIT; ++k) s += cpart[k * m + j];
    c = s * log(s / (double)b[j] + 1e-16);
  }
  if (rows_on) for (int64_t i = j; i < n; i += (int64_t)gridDim.x * 128) r += krow[i];
  c = block_sum_fixed(c);
  r = block_sum_fixed(r);
  if (threadIdx.x == 0) { slots[2 * blockIdx.x] = r; slots[2 * blockIdx.x + 1] = c; }
}

// cost, and cost + reg * (the plan's KL or entropy) + the marginal penalties.
template <typename T>
__global__ void __launch_bounds__(256) unb_total_kernel(const double* slots, int blocks, const double* vals, double reg, double rm1,
                                                        double rm2, int rows_on, int cols_on, T* out) {
  double r = 0.0, c = 0.0;
  for (int k = threadIdx.x; k < blocks; k += 256) { r += slots[2 * k]; c += slots[2 * k + 1]; }
  r = block_sum_fixed(r);
  c = block_sum_fixed(c);
  if (threadIdx.x == 0) {
    double t = vals[0] + reg * vals[1];
    if (rows_on) t += rm1 * r;
    if (cols_on) t += rm2 * c;
    out[0] = (T)vals[0];
    out[1] = (T)t;
  }
}

}  // namespace otg

using namespace otg;

extern "C" {

int otg_unbalanced_vectors(int dtype, int64_t n, int64_t m, const void* u, const void* v, const void* alw, const void* bew, void* ut,
                           void* vt, void* lu, void* lv, cudaStream_t stream) {
  if (!u || !v || !ut || !vt || !lu || !lv || n < 1 || m < 1) return OTG_ERR_ARG;
  if (dtype != OTG_F32 && dtype != OTG_F64) return OTG_ERR_DTYPE;
  const int64_t blocks = (n + m + 255) / 256;
  if (blocks > INT32_MAX) return OTG_ERR_UNSUPPORTED;
  auto run = [&](auto z) {
    using T = decltype(z);
    unb_vectors_kernel<T><<<(unsigned)blocks, 256, 0, stream>>>(n, m, static_cast<const T*>(u), static_cast<const T*>(v),
                                                                static_cast<const T*>(alw), static_cast<const T*>(bew),
                                                                static_cast<T*>(ut), static_cast<T*>(vt), static_cast<T*>(lu),
                                                                static_cast<T*>(lv));
  };
  if (dtype == OTG_F64) run(0.0); else run(0.f);
  return cudaGetLastError() == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}

int64_t otg_unbalanced_total_doubles(int64_t n, int64_t m) { return n + UB_SPLIT * m + 2 * ((m + 127) / 128); }

int otg_unbalanced_total(int dtype, const void* P, int64_t n, int64_t m, int64_t ldp, const void* a, const void* b, const double* vals,
                         double reg, double reg_m1, double reg_m2, double* scratch, void* out, cudaStream_t stream) {
  if (!P || !a || !b || !vals || !scratch || !out || n < 1 || m < 1 || ldp < m) return OTG_ERR_ARG;
  if (dtype != OTG_F32 && dtype != OTG_F64) return OTG_ERR_DTYPE;
  const int rows_on = !isinf(reg_m1), cols_on = !isinf(reg_m2);
  const int64_t rb = (n + 7) / 8, cb = (m + 127) / 128;
  if (rb + cb * UB_SPLIT > INT32_MAX) return OTG_ERR_UNSUPPORTED;
  double *krow = scratch, *cpart = krow + n, *slots = cpart + UB_SPLIT * m;
  auto run = [&](auto z) {
    using T = decltype(z);
    if (rows_on || cols_on)
      unb_marginals_kernel<T><<<(unsigned)(rb + (cols_on ? cb * UB_SPLIT : 0)), 256, 0, stream>>>(
          static_cast<const T*>(P), n, m, ldp, static_cast<const T*>(a), rows_on, rb, krow, cpart);
    unb_terms_kernel<T><<<(unsigned)cb, 128, 0, stream>>>(n, m, static_cast<const T*>(b), rows_on, cols_on, krow, cpart, slots);
    unb_total_kernel<T><<<1, 256, 0, stream>>>(slots, (int)cb, vals, reg, reg_m1, reg_m2, rows_on, cols_on, static_cast<T*>(out));
  };
  if (dtype == OTG_F64) run(0.0); else run(0.f);
  return cudaGetLastError() == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}

}  // extern "C"
