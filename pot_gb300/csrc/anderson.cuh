// Anderson mixing of a Sinkhorn potential update, one CTA per problem.
//
// The map F(v) = colT(rowT(v)) (a row update followed by a column update)
// has the Sinkhorn potentials as fixed points.  With depth D the v of the
// next row update is  sum_k alpha_k F(v_k)  over the last D iterates, alpha
// minimising |sum_k alpha_k (F(v_k) - v_k)|_2 with sum alpha = 1: the normal
// equations of the residual Gram matrix with a Tikhonov term 1e-10 trace / D,
// solved by Gaussian elimination with partial pivoting; a failed solve, or
// one with sum |alpha| >= 1e4, restarts the history and takes the plain step.
// No reference counterpart (the warm-start refinement); the caller's stop
// test is unchanged.
#pragma once
#include "common.cuh"
#include "../../include/pot_gb300.h"

namespace otg {

constexpr double AND_LAMBDA = 1e-10;   // Tikhonov term, relative to trace / D
constexpr double AND_MAX_L1 = 1e4;     // larger sum |alpha|: restart with the plain step

// The weights of the mixed iterate, by one warp: lane q < nh brings the dot
// <r_new, R_q> and gets the weight of slot q.  Updates G; false: take the
// plain step.
//
// (G + lambda I) w = 1 by Gauss-Jordan elimination with partial pivoting, a
// row per lane (rows beyond nh are those of the identity).  A chain of
// latencies: an FP64 division takes about 0.5 us here, so there is one per
// pivot and two more (elimination with back substitution by the warp: 25 of
// them, 27 us for a step; by one thread 60 us).
__device__ __forceinline__ bool anderson_solve(int D, int nh, int s, double dot, double* G, int lane, double& w) {
  constexpr int MD = OTG_ANDERSON_MAX_DEPTH;
  double row[MD + 1], dots[MD];
#pragma unroll
  for (int j = 0; j < MD; ++j) dots[j] = __shfl_sync(0xffffffffu, dot, j);
  if (lane < nh) {
#pragma unroll
    for (int j = 0; j < MD; ++j) row[j] = j < nh ? (lane == s ? dots[j] : j == s ? dot : __ldcg(G + lane * D + j)) : 0.0;
    G[s * D + lane] = dot;
    G[lane * D + s] = dot;
  } else {
#pragma unroll
    for (int j = 0; j < MD; ++j) row[j] = j == lane ? 1.0 : 0.0;
  }
  row[MD] = lane < nh ? 1.0 : 0.0;
  double diag = 0.0;
#pragma unroll
  for (int j = 0; j < MD; ++j) if (j == lane) diag = row[j];
  double tr = 0.0;
  for (int i = 0; i < nh; ++i) tr += __shfl_sync(0xffffffffu, diag, i);
  const double lam = AND_LAMBDA * tr / nh;
#pragma unroll
  for (int j = 0; j < MD; ++j) if (j == lane && lane < nh) row[j] += lam;
  bool ok = nh > 1 && tr > 0.0;
#pragma unroll
  for (int c = 0; c < MD; ++c) {
    if (c < nh) {
      // the first of the largest entries of the column at or below the diagonal
      double best = lane >= c && lane < nh ? fabs(row[c]) : -1.0;
      int piv = lane;
#pragma unroll
      for (int o = 1; o < MD; o *= 2) {
        const double x = __shfl_xor_sync(0xffffffffu, best, o);
        const int y = __shfl_xor_sync(0xffffffffu, piv, o);
        if (x > best || (x == best && y < piv)) { best = x; piv = y; }
      }
      best = __shfl_sync(0xffffffffu, best, 0);
      piv = __shfl_sync(0xffffffffu, piv, 0);
      if (!(best > 0.0)) { ok = false; piv = c; }
      const int from = lane == c ? piv : lane == piv ? c : lane;
      double top[MD + 1];
#pragma unroll
      for (int j = 0; j <= MD; ++j) {
        if (j >= c) {
          row[j] = __shfl_sync(0xffffffffu, row[j], from);
          top[j] = __shfl_sync(0xffffffffu, row[j], c);
        }
      }
      if (lane != c && lane < nh && ok) {
        const double f = row[c] / top[c];
#pragma unroll
        for (int j = 0; j <= MD; ++j) if (j > c) row[j] -= f * top[j];
      }
    }
  }
  double x = 0.0;
#pragma unroll
  for (int j = 0; j < MD; ++j) if (j == lane && lane < nh) x = row[MD] / row[j];
  double sw = 0.0, l1 = 0.0;
#pragma unroll
  for (int i = MD - 1; i >= 0; --i) sw += __shfl_sync(0xffffffffu, x, i);
  w = x / sw;
#pragma unroll
  for (int i = 0; i < MD; ++i) l1 += fabs(__shfl_sync(0xffffffffu, w, i));
  return ok && isfinite(l1) && l1 < AND_MAX_L1;
}

// One problem's step, called by every thread of the CTA.  vold: v_k, vnew:
// F(v_k) on entry and the mixed v on return, both at column offset `co`
// (m columns); F and R: D history slots of stride `stride` (slot-major);
// G: the problem's D x D residual Gram matrix; cnt: iterates taken so far.
template <typename T>
__device__ void anderson_step(int D, int m, int64_t co, int64_t stride, const T* vold, T* vnew, T* F, T* R,
                              double* G, int32_t* cnt_p) {
  constexpr int MD = OTG_ANDERSON_MAX_DEPTH;
  __shared__ double s_dot[MD];
  __shared__ double s_alpha[MD];
  __shared__ int s_keep;
  const int cnt = __ldcg(cnt_p);
  const int s = cnt % D;                       // slot of the new iterate
  const int nh = cnt + 1 < D ? cnt + 1 : D;    // slots in use after the insert
  // insert, and this thread's share of the dots <r_new, R_q>
  double acc[MD];
#pragma unroll
  for (int q = 0; q < MD; ++q) acc[q] = 0.0;
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    const T f = __ldcg(vnew + co + j);
    const T r = f - __ldcg(vold + co + j);
    F[(int64_t)s * stride + co + j] = f;
    R[(int64_t)s * stride + co + j] = r;
#pragma unroll
    for (int q = 0; q < MD; ++q) {
      if (q < nh) {
        const T rq = q == s ? r : __ldcg(R + (int64_t)q * stride + co + j);
        acc[q] += widen(r) * widen(rq);
      }
    }
  }
  // all dots at once: a halving butterfly over the warp (lane l ends with dot
  // l / 4), then the warps in order.  FP64 issues at two lanes per clock, so
  // eight separate block sums were a third of the step.
  {
    __shared__ double s_part[32][MD];
    int o = 16;
#pragma unroll
    for (int h = MD / 2; h >= 1; h /= 2) {
      const bool up = threadIdx.x & o;
#pragma unroll
      for (int q = 0; q < h; ++q) {
        const double keep = up ? acc[q + h] : acc[q], give = up ? acc[q] : acc[q + h];
        acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      o >>= 1;
    }
    double d = acc[0];
    for (int q = 16 / MD; q > 0; q >>= 1) d += __shfl_xor_sync(0xffffffffu, d, q);
    __syncthreads();
    if ((threadIdx.x & 31) % (32 / MD) == 0) s_part[threadIdx.x >> 5][(threadIdx.x & 31) / (32 / MD)] = d;
    __syncthreads();
    if (threadIdx.x < MD) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w][threadIdx.x];
      s_dot[threadIdx.x] = t;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    double w;
    const bool ok = anderson_solve(D, nh, s, lane < MD ? s_dot[lane] : 0.0, G, lane, w);
    if (lane < MD) s_alpha[lane] = w;
    if (lane == 0) {
      // a first iterate, or a failed solve: the plain step; after a failure
      // the history restarts with the next iterate
      s_keep = ok;
      *cnt_p = ok || nh == 1 ? cnt + 1 : 0;
    }
  }
  __syncthreads();
  if (s_keep) {
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
      double vm = 0.0;
      for (int q = 0; q < nh; ++q) vm += s_alpha[q] * widen(__ldcg(F + (int64_t)q * stride + co + j));
      vnew[co + j] = (T)vm;
    }
  }
  // after a restart vnew keeps F(v_k): the plain step
  __syncthreads();
}

}  // namespace otg
