// Gradients of the Sinkhorn loss sum(M * P) at the solution, by implicit
// differentiation (the system and its gauge are stated in
// pot_gb300/_autograd.py): with r = (M o P) 1, c = (M o P)^T 1,
//   (diag(b) - P^T diag(1/a) P + b b^T / sum(b)) mu = c - P^T (r / a)
// by conjugate gradients preconditioned with diag(b), then
//   lam = (r - P mu) / a,  t = b . mu / sum(b),
//   dM = P o (1 + (lam + mu - M) / reg),  da = lam + t,  db = mu - t.
// No counterpart in the reference, which differentiates through its iterations
// (ot/bregman/_sinkhorn.py:435-438 on the torch backend).
//
// One persistent cooperative launch.  P^T diag(1/a) P p is one read of P, as
// an iteration of the dense solver is one read of the cost: a row's dot
// product with p, divided by a, scales the same entries into the column sums
// (fused_impl.cuh, whose row split and hand-over this uses).  Each CTA keeps
// p, mu, the residual and S p whole in shared memory and takes the scalar
// steps by itself, in the same order as every other, so an iteration has two
// hand-overs and no reduction over the grid.  n = m = 500: eight iterations;
// as torch operations with a host decision per iteration the backward pass
// took 3.9 ms, 0.7 ms of it on the device.
#include "fused_impl.cuh"

namespace otg {

constexpr int GR_MAXM = 4096;  // four vectors of this many doubles in shared memory

struct GradArgs {
  FusedArgs<double> F;         // M holds P; a, b; published words; split
  const double* M; int64_t ldmM;
  double reg, rtol;
  int max_iter;
  double *r;                   // [n] (M o P) 1
  double *gM, *ga, *gb; int64_t ldg;
};

// Block sums of three values; every thread gets them.
__device__ __forceinline__ void gr_sum3(double (&x)[3], double (*scr)[FU_WARPS]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) x[q] = warp_sum(x[q]);
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < 3; ++q) scr[q][threadIdx.x >> 5] = x[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double t = 0.0;
    for (int w = 0; w < FU_WARPS; ++w) t += scr[q][w];
    x[q] = t;
  }
}

// One pass over the CTA's rows.  STEP 0: right-hand side (rows of M o P);
// STEP 1: P^T diag(1/a) P p; STEP 2: the gradients.
template <int NK, int STEP>
__device__ __forceinline__ void gr_pass(const GradArgs& G, const FuRow& R, const FuSmem<double>& sm,
                                        double (*red)[FU_WARPS][fu_rb(NK)], double t_gauge, unsigned ep) {
  using V = FuV<double>;
  constexpr int RB = NK > 4 ? 1 : fu_rb(NK) / 2, LPR = 32 / RB, W = 2;  // half a batch: STEP 0 and 2 hold M as well
  const FusedArgs<double>& A = G.F;
  V acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = V::zero();
  int par = 0;
  const int myrow = R.lane / LPR;
  for (int rb = R.ga; rb < R.gb; rb += RB) {
    const int nr = min(RB, R.gb - rb);
    double x[RB][NK][W], s[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const int row = rb + min(q, nr - 1);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int col = (k * R.gt + R.tg) * W;
        x[q][k][0] = x[q][k][1] = 0.0;
        if (col < A.mv) fu_get_global(A, row, col, 0.0, x[q][k]);
      }
    }
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const int row = rb + min(q, nr - 1);
      s[q] = 0.0;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int col = (k * R.gt + R.tg) * W;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          if (STEP == 0) {
            const double mp = col + w < A.m ? x[q][k][w] * G.M[(int64_t)row * G.ldmM + col + w] : 0.0;
            s[q] += mp;
            if (q < nr) { if (w == 0) acc[k].a += mp; else acc[k].b += mp; }
          } else {
            s[q] = fma(x[q][k][w], sm.vs[col + w], s[q]);
          }
        }
      }
    }
    // (the scratch is sized for a whole batch)
    const double t = fu_group<double, RB, false>(s, R, A.G, red, par);
    const int row = min(rb + myrow, R.gb - 1);
    const double ai = A.a[row], ia = ai > 0.0 ? 1.0 / ai : 0.0;
    double f;  // what the row's entries are scaled with; STEP 2: lam
    if (STEP == 0) {
      f = -ia * t;
      if (R.tg < 32 && R.lane % LPR == 0 && myrow < nr) G.r[row] = t;
    } else if (STEP == 1) {
      f = ia * t;
    } else {
      f = (G.r[row] - t) * ia;
      if (R.tg < 32 && R.lane % LPR == 0 && myrow < nr) G.ga[row] = f + t_gauge;
    }
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const double fq = __shfl_sync(0xffffffffu, f, q * LPR);
      if (q < nr) {
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const int col = (k * R.gt + R.tg) * W;
          if (STEP < 2) {
            acc[k].a = fma(x[q][k][0], fq, acc[k].a);
            acc[k].b = fma(x[q][k][1], fq, acc[k].b);
          } else {
#pragma unroll
            for (int w = 0; w < W; ++w)
              if (col + w < A.m)
                G.gM[(int64_t)(rb + q) * G.ldg + col + w] =
                    x[q][k][w] * (1.0 + (fq + sm.vs[col + w] - G.M[(int64_t)(rb + q) * G.ldmM + col + w]) / G.reg);
          }
        }
      }
    }
  }
  if (STEP < 2) fu_publish_cols<double, NK>(A, R, sm, acc, ep);
}

template <int NK>
__global__ void __launch_bounds__(FU_THREADS, 1) sinkhorn_grad_kernel(const __grid_constant__ GradArgs G) {
  extern __shared__ __align__(16) unsigned char gr_smem[];
  __shared__ double red[2][FU_WARPS][fu_rb(NK)];
  __shared__ double s_s[FU_WARPS * 32], scr[3][FU_WARPS];
  const FusedArgs<double>& A = G.F;
  FuRow R{};
  R.r0 = (int)((int64_t)A.n * blockIdx.x / gridDim.x);
  R.r1 = (int)((int64_t)A.n * (blockIdx.x + 1) / gridDim.x);
  R.warp = threadIdx.x >> 5;
  R.lane = threadIdx.x & 31;
  R.NG = FU_WARPS / A.G;
  R.g = R.warp / A.G;
  R.gt = A.G * 32;
  R.tg = threadIdx.x - R.g * R.gt;
  {
    const int rows = R.r1 - R.r0, per = (rows + R.NG - 1) / R.NG;
    R.live = (rows + per - 1) / per;
    R.ga = min(R.r1, R.r0 + per * R.g);
    R.gb = min(R.r1, R.ga + per);
  }
  FuSmem<double> sm{}, sp{};
  sm.vs = reinterpret_cast<double*>(gr_smem);      // p, then mu
  sp.vs = sm.vs + A.mp;                            // S p
  double* mu = sp.vs + A.mp;
  double* res = mu + A.mp;
  sm.buf = res + A.mp;
  const int cb = (int)((int64_t)A.m * blockIdx.x / gridDim.x), ce = (int)((int64_t)A.m * (blockIdx.x + 1) / gridDim.x);
  unsigned gen = 0;
  for (int j = cb + threadIdx.x; j < ce; j += FU_THREADS) A.vll[2 * j] = A.vll[2 * j + 1] = 0ull;
  for (int j = threadIdx.x; j < 2 * A.m; j += FU_THREADS) A.part[(int64_t)blockIdx.x * A.m * 2 + j] = 0ull;
  if (threadIdx.x == 0) A.stll[blockIdx.x] = 0ull;
  for (int j = threadIdx.x; j < A.mp; j += FU_THREADS) sm.vs[j] = sp.vs[j] = mu[j] = res[j] = 0.0;
  if (!fu_barrier(A.bar, gen, A.info + 3, A.timeout_ns)) return;

  unsigned ep = 1;
  double e2 = 0.0;
  gr_pass<NK, 0>(G, R, sm, red, 0.0, ep);
  bool ok = fu_merge<double>(A, R, s_s, ep, [&](int j, double s) { Ll<double>::put(A.vll + 2 * j, s, ep); });
  if (__syncthreads_or(!ok)) ok = false;
  if (threadIdx.x == 0) ll_st(A.stll + blockIdx.x, 0, ep);
  if (fu_collect(A, sp, ep, false, ok, e2) & FU_ABORT) return;  // sp: the right-hand side
  // mu = 0, residual = right-hand side, p = z = residual / b
  double d[3] = {0.0, 0.0, 0.0}, sb = 0.0;
  for (int j = threadIdx.x; j < A.m; j += FU_THREADS) {
    const double bj = A.b[j], x = sp.vs[j], z = bj > 0.0 ? x * (1.0 / bj) : 0.0;
    res[j] = x;
    sm.vs[j] = z;
    d[0] = fma(x, z, d[0]); d[1] = fma(x, x, d[1]); d[2] = fma(bj, z, d[2]);
    sb += bj;
  }
  gr_sum3(d, scr);
  double rz = d[0], rr = d[1], bp = d[2];
  double sb3[3] = {sb, 0.0, 0.0};
  gr_sum3(sb3, scr);
  sb = sb3[0];
  const double stop = (G.rtol * sqrt(rr)) * (G.rtol * sqrt(rr)), beta = 1.0 / sb;
  for (int it = 0; it < G.max_iter && !(rr <= stop); ++it) {
    ++ep;
    __syncthreads();  // p is whole
    gr_pass<NK, 1>(G, R, sm, red, 0.0, ep);
    ok = fu_merge<double>(A, R, s_s, ep, [&](int j, double s) {
      const double bj = A.b[j];
      Ll<double>::put(A.vll + 2 * j, bj * sm.vs[j] - s + (beta * bp) * bj, ep);
    });
    if (__syncthreads_or(!ok)) ok = false;
    if (threadIdx.x == 0) ll_st(A.stll + blockIdx.x, 0, ep);
    if (fu_collect(A, sp, ep, false, ok, e2) & FU_ABORT) return;
    d[0] = d[1] = d[2] = 0.0;
    for (int j = threadIdx.x; j < A.m; j += FU_THREADS) d[0] = fma(sm.vs[j], sp.vs[j], d[0]);
    gr_sum3(d, scr);
    if (!(d[0] > 0.0)) break;
    const double alpha = rz / d[0];
    d[0] = d[1] = d[2] = 0.0;
    for (int j = threadIdx.x; j < A.m; j += FU_THREADS) {
      mu[j] = fma(alpha, sm.vs[j], mu[j]);
      const double x = fma(-alpha, sp.vs[j], res[j]);
      res[j] = x;
      const double bj = A.b[j], z = bj > 0.0 ? x * (1.0 / bj) : 0.0;
      sp.vs[j] = z;
      d[0] = fma(x, z, d[0]); d[1] = fma(x, x, d[1]); d[2] = fma(bj, z, d[2]);
    }
    gr_sum3(d, scr);
    const double g = d[0] / rz;
    for (int j = threadIdx.x; j < A.m; j += FU_THREADS) sm.vs[j] = fma(g, sm.vs[j], sp.vs[j]);
    rz = d[0];
    rr = d[1];
    bp = fma(g, bp, d[2]);
  }
  __syncthreads();
  d[0] = d[1] = d[2] = 0.0;
  for (int j = threadIdx.x; j < A.m; j += FU_THREADS) {
    d[0] = fma(A.b[j], mu[j], d[0]);
    sm.vs[j] = mu[j];
  }
  gr_sum3(d, scr);  // (its barriers make mu whole for the pass)
  const double t = d[0] / sb;
  gr_pass<NK, 2>(G, R, sm, red, t, 0);
  for (int j = cb + threadIdx.x; j < ce; j += FU_THREADS) G.gb[j] = mu[j] - t;
}

namespace {

struct GradPlan { int grid, G, NK, mp, buf; size_t smem, part, vll, stll, ell, r, ctl, total; };

bool grad_plan(int64_t n, int64_t m, GradPlan& f) {
  const FuDevice d = fu_device();
  if (n < 1 || m < 1 || m > GR_MAXM || n > 0x7fffff00 || d.sms < 1) return false;
  const int64_t V = (m + 1) / 2;
  f.grid = fu_grid<double>(n, m, 0, d.sms);
  f.NK = 1;
  while (f.NK < 8 && (int64_t)FU_WARPS * 32 * f.NK < V) f.NK *= 2;
  f.G = 1;
  while (f.G < FU_WARPS && (int64_t)f.G * 32 * f.NK < V) f.G *= 2;
  f.mp = f.NK * f.G * 32 * 2;
  const int NG = FU_WARPS / f.G;
  f.buf = NG > 1 ? NG * f.mp : 0;
  f.smem = sizeof(double) * (4 * (size_t)f.mp + f.buf);
  size_t off = 0;
  auto take = [&](size_t b) { const size_t o = off; off += (b + 255) / 256 * 256; return o; };
  f.part = take(16 * (size_t)f.grid * m);
  f.vll = take(16 * (size_t)m);
  f.stll = take(8 * (size_t)f.grid);
  f.ell = take(96 * (size_t)f.grid);
  f.r = take(8 * (size_t)n);
  f.ctl = take(256);
  f.total = off;
  return f.smem + 8192 <= d.smem;
}

template <int NK>
int grad_start(GradArgs& G, const GradPlan& f, cudaStream_t st) {
  const void* k = (const void*)sinkhorn_grad_kernel<NK>;
  if (!allow_smem(k, f.smem)) return OTG_ERR_CUDA;
  void* args[] = {&G};
  return cudaLaunchCooperativeKernel(k, dim3(f.grid), dim3(FU_THREADS), args, f.smem, st) == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}

}  // namespace
}  // namespace otg

using namespace otg;

extern "C" {

size_t otg_sinkhorn_grad_workspace_bytes(int64_t n, int64_t m) {
  GradPlan f;
  return grad_plan(n, m, f) ? f.total : 0;
}

int otg_sinkhorn_grad(const double* P, int64_t ldp, const double* M, int64_t ldm, int64_t n, int64_t m, const double* a,
                      const double* b, double reg, double rtol, int32_t max_iter, double* gM, int64_t ldg, double* ga, double* gb,
                      void* workspace, size_t workspace_bytes, int32_t* info, cudaStream_t stream) {
  if (!P || !M || !a || !b || !gM || !ga || !gb || !workspace || !info || n < 1 || m < 1 || ldp < m || ldm < m || ldg < m ||
      max_iter < 0)
    return OTG_ERR_ARG;
  GradPlan f;
  if (!grad_plan(n, m, f)) return OTG_ERR_UNSUPPORTED;
  if (workspace_bytes < f.total) return OTG_ERR_WORKSPACE;
  char* w = static_cast<char*>(workspace);
  GradArgs G{};
  G.F.M = P; G.F.ldm = ldp; G.F.n = (int)n; G.F.m = (int)m;
  G.F.mv = (int)((m + 1) / 2 * 2);
  G.F.gvec = m % 2 == 0 && ldp % 2 == 0 && (uintptr_t)P % 16 == 0;
  G.F.a = a; G.F.b = b;
  G.F.part = reinterpret_cast<unsigned long long*>(w + f.part);
  G.F.vll = reinterpret_cast<unsigned long long*>(w + f.vll);
  G.F.stll = reinterpret_cast<unsigned long long*>(w + f.stll);
  G.F.ell = reinterpret_cast<unsigned long long*>(w + f.ell);
  G.F.info = info;
  G.F.bar = reinterpret_cast<unsigned*>(w + f.ctl);
  G.F.timeout_ns = 4000000000ull;
  G.F.G = f.G; G.F.kv = f.NK; G.F.mp = f.mp; G.F.buf_elems = f.buf;
  G.M = M; G.ldmM = ldm; G.reg = reg; G.rtol = rtol; G.max_iter = max_iter;
  G.r = reinterpret_cast<double*>(w + f.r);
  G.gM = gM; G.ga = ga; G.gb = gb; G.ldg = ldg;
  if (cudaMemsetAsync(w + f.ctl, 0, 256, stream) != cudaSuccess) return OTG_ERR_CUDA;
  if (cudaMemsetAsync(info, 0, 4 * sizeof(int32_t), stream) != cudaSuccess) return OTG_ERR_CUDA;
  switch (f.NK) {
    case 1: return grad_start<1>(G, f, stream);
    case 2: return grad_start<2>(G, f, stream);
    case 4: return grad_start<4>(G, f, stream);
    default: return grad_start<8>(G, f, stream);
  }
}

}  // extern "C"
