// Shared pieces of the batch kernels (multi.cu, multi_fused.cuh).
#pragma once
#include "common.cuh"
#include "anderson.cuh"
#include "../../include/pot_gb300.h"

namespace otg {

// 256 threads at no more than 64 registers, four CTAs per SM (float): the
// loads in flight come from the 32 resident warps (measured: 0.79 of the copy peak
// against 0.71 for two CTAs of 118 registers with loads software-pipelined
// one group ahead, on 512 cost blocks of 2048 x 2048).
constexpr int MT_THREADS = 256;
// CTAs per SM: float at 64 registers; double keeps 128 registers (no spills)
template <typename T> struct MtBlocks { static constexpr int value = sizeof(T) == 4 ? 4 : 2; };
constexpr int MT_RW = 4;       // rows per warp in the row pass
constexpr int MT_GCOL = 4;     // rows folded per max update (column pass)

template <typename T> struct MPair { T mx, s; };

template <typename T>
struct MultiArgs {
  const T* M; const int64_t* m_off; const int32_t* rows; const int32_t* cols; const int32_t* ldm;
  const int64_t* r_off; const int64_t* c_off;
  const T* a; const T* b; const T* warm_u;
  const double* reg;
  int32_t nprob, max_iter;
  double stop_thr;
  // per-problem decomposition: partial buffers sized for nsr_max row chunks;
  // the split in use (nsr, rchunk) is chosen at every rebuild of the active
  // list from the amount of work left
  const int32_t* nsr_max;
  int32_t* nsr;             // row chunks (column pass), device-chosen
  int32_t* rchunk;          // rows per chunk, device-chosen
  const int64_t* pc_off;    // offset of problem's partials [nsr_max][m]
  // state
  T* u; T* v0; T* v1;       // base-2 potentials, packed like a / b
  MPair<T>* pcol;
  double* err2;             // per problem: squared error of the last check (joint stop)
  double* e2col;            // per column: squared marginal error (check passes), packed like b
  bool joint;               // whole-batch stop on the largest error
  // Anderson mixing of the v update (depth 0: off): history slots of F(v)
  // and of the residual F(v) - v, [depth][total_cols] each (slot-major,
  // packed like b), residual Gram matrices [nprob][depth][depth] and the
  // number of iterates taken so far per problem
  int and_depth;
  int64_t total_cols;
  T* and_F; T* and_R;
  double* and_G;
  int32_t* and_cnt;
  int32_t* active;          // active problem ids [nprob]
  int64_t* ucol_pre;        // prefix of column-pass units over the active list [nprob+1]
  int64_t* urow_pre;        // prefix of row-pass units
  int64_t* colpre;          // prefix of columns (merge) over the active list
  int32_t* ctl;             // [0] n active, [1] abort
  int32_t* leave_cnt;       // [2] problems leaving at a decision (alternate decisions)
  unsigned* bar;
  // outputs
  T* out_u; T* out_v;
  int32_t* status; int32_t* niter; double* err;
  uint64_t timeout_ns;
  T omega;                  // over-relaxation (1: plain)
  bool relax;
  int period;               // iterations between stop tests
  int upw, cap_fill, cap_tail;  // schedule: units per warp, row-split caps
  // tail handoff: most problems handed over (0: never), CTAs per cluster,
  // shared-memory bytes for one CTA's rows of a cost block
  int tail_max, tail_cl;
  int64_t tail_tile;
  // one-read kernel (multi_fused.cuh): warps per row, ring chunks per worker,
  // columns of a worker's v, widest block; column sums and (maximum, sum)
  // pairs of the workers; per problem: column sums too small to trust
  int fG, fNK, fNC, fmp, fmm;
  T* fpart; T* fpairs;
  int32_t* fbad;
  int32_t* flim;            // per problem: exponent below which a column sum cannot be trusted
  double* and_part; double* and_w;  // dots of the blocks of 32 columns, weights of the problems (mf_anderson)
};

// Tail kernel limits: columns, rows per CTA
constexpr int TL_MAXM = 2048;
constexpr int TL_MAXR = 1024;
constexpr int TL_THREADS = 256;

// Index of the active slot whose prefix range holds `unit` (pre[k] <= unit < pre[k+1]).
__device__ __forceinline__ int mt_find(const int64_t* pre, int n, int64_t unit) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldcg(pre + mid) <= unit) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Slot cursor over a prefix array: pre[k] <= item < pre[k+1].  Items visited
// in increasing order mostly stay in the slot or move to the next one, so the
// binary search (a chain of dependent L2 loads) runs about once per problem.
struct MtSlot {
  int k = -1;
  int64_t lo = 0, hi = 0;
  __device__ __forceinline__ bool seek(const int64_t* pre, int n, int64_t item) {
    if (k >= 0 && item >= lo && item < hi) return false;
    if (k >= 0 && item >= hi && k + 1 < n && __ldcg(pre + k + 2) > item) ++k;
    else k = mt_find(pre, n, item);
    lo = __ldcg(pre + k);
    hi = __ldcg(pre + k + 1);
    return true;
  }
};

// Contiguous share [beg, end) of `total` items for worker w of nw.
__device__ __forceinline__ void mt_share(int64_t total, long w, long nw, int64_t& beg, int64_t& end) {
  beg = total * w / nw;
  end = total * (w + 1) / nw;
}

// Anderson step (one CTA per active problem, anderson.cuh): the new v of
// every active problem is mixed over its history.  Kept out of line, like
// the joint decision: it must not weigh on the registers of the passes.
template <typename T>
__device__ __noinline__ void mt_anderson(const MultiArgs<T>& A, int nact, const T* vcur, T* vnxt) {
  for (int k = blockIdx.x; k < nact; k += gridDim.x) {
    const int p = __ldcg(A.active + k);
    anderson_step<T>(A.and_depth, A.cols[p], A.c_off[p], A.total_cols, vcur, vnxt, A.and_F, A.and_R,
                     A.and_G + (int64_t)p * A.and_depth * A.and_depth, A.and_cnt + p);
  }
}

// Largest error of the active problems from err2 (a max: the same in any
// order); every thread gets it.  Kept out of line: it runs once per check and
// its registers must not weigh on the passes.
template <typename T>
__device__ __noinline__ double mt_joint_largest(const MultiArgs<T>& A, int nact) {
  __shared__ double s_mx[MT_THREADS / 32];
  double mx = 0.0;
  for (int k = threadIdx.x; k < nact; k += blockDim.x) {
    const double e2 = __ldcg(A.err2 + __ldcg(A.active + k));
    mx = isnan(e2) ? (double)INFINITY : fmax(mx, e2);  // a NaN error never meets the test
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, s_mx[w]);
  __syncthreads();
  return sqrt(mx);
}

// The one-read kernel for this batch (fields f* and G, NC, NK set by
// multi_fused_plan); multi_fused_f32.cu, multi_fused_f64.cu.
struct MultiFusedPlan { int G, NK, NC, mp; size_t smem; };
bool multi_fused_plan(int dtype, int max_ldm, size_t smem_max, MultiFusedPlan& f);
int multi_fused_launch(const MultiArgs<float>& A, bool logf, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st);
int multi_fused_launch(const MultiArgs<double>& A, bool logf, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st);

}  // namespace otg
