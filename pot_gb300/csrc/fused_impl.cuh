// Dense Sinkhorn with ONE read of the cost per iteration, one persistent
// cooperative launch per solve (scaling, log and unbalanced forms; the
// iterations, stop tests and reverts are those of dense.cu).
//
// Once the row update of row i is known, the row's share of the NEXT column
// update follows from the same entries: with e_ij = exp(x_ij + v_j + shift)
// and s_i = sum_j e_ij the updated plan row is P_ij = e_ij a_i / s_i, and
// sum_i P_ij is both the column marginal of the stop test and all that the
// column update needs, v_j += log(b_j / sum_i P_ij).  So an iteration is
//   pass   every CTA goes over its own rows: row reduction, row update, then
//          the scaled entries (still in registers) are added to per-thread
//          column sums, which go to the CTA's slot
//   merge  every CTA adds up the slots of its share of the columns in slot
//          order, updates v and the squared marginal error
// with one exponential per entry instead of two and half the HBM traffic of
// a column pass followed by a row pass.
//
// Hand-over.  A grid barrier costs about 1.7 us here (fence, atomic and poll:
// three trips to L2) and the loads behind it one more trip, so the column
// sums and the new v do not go through barriers: each value is stored in one
// 64-bit word with the iteration number (a float64 in two such words) and the
// reader polls the value itself.  A slot of column sums is rewritten only
// after its writer has read all of the next v and the flags, to which every
// reader of the slot has contributed by then.  v, the per-iteration flags and
// the error shares, which travel the same way so that every CTA takes the same
// decisions, are rewritten only behind the merge, and nobody leaves the merge
// before it has seen column sums of the iteration from every CTA, which a CTA
// publishes when it is done with all three: single buffers are enough.  (With
// more CTAs than columns some have no column to merge.  They wait for the
// first column's sums like the CTA that owns it; without that nothing stood
// between reading the flags of one iteration and writing those of the next.)
//
// Split.  A CTA of 8 warps (255 registers a thread: nothing may spill, as the
// shared memory leaves an L1 of 28 KB and a spilled loop runs at L2 latency;
// measured 1.5 to 2 times slower) owns a contiguous range of rows; G warps
// share a row and 8 / G groups work side by side.  A thread holds NK 16-byte
// vectors of each of RB rows, at most 256 bytes of entries.
//   Resident: the CTA's rows stay in shared memory for the whole solve; the
//   fewest vectors per thread (NK) that cover a row and let the rows fit, so
//   that up to 8 rows share one reduction (reduce-scatter over the warp, one
//   barrier), one division and one read of v.
//   Streamed (cost larger than the SMs' shared memory, 30 MB): NK = 10 to 16,
//   the even number that covers the row with the fewest groups' threads, one
//   row at a time per group, so that one group's reduction overlaps another's
//   exponentials.  A ring of bulk copies issued by one lane per group, in
//   chunks of half a row; 120 to 200 KB are in flight per SM, and the copies
//   of the next pass's first rows cross the hand-over.
//
// Range of the shortcut.  Log form: the shift of row i is its previous
// potential less log a_i, so e_ij is the row's previous plan entry over a_i
// and s_i is near one; rows whose s_i leaves [2^-30, 2^30] (first iterations
// from a far start, non-finite input) take the running-maximum form on the
// same entries.  Rows of no weight have a shift of -inf: their entries are
// zeros, their potential -inf.  (With a shift of u - log a they were not
// numbers and went through the running maxima with the rows of their batch:
// half of the rows empty, 8192^2 float32 98 us per iteration, now 59.)  What can be lost in a column sum are entries
// below 2^-126 (2^-1074 in float64) times the row factors a_i / s_i, together
// 2^-96 (2^-1044) of the mass.  A column sum that is not 2^26 (2^59) times
// that is recomputed in that iteration with running maxima: one more pass over
// such columns and two grid barriers.  (Bounds that know neither the type nor
// the mass, and a pass over all columns, made Gaussian histograms, whose tails
// meet them in every iteration, slower than two passes: 8192^2 float32 278 us
// per iteration, two passes 95; 3000 x 1100 float64 439, two passes 845.)
//
// float64 log form, cost resident: this GPU issues FP64 at about two lanes
// per clock and SM, and an exponential costs some ten such operations.
// The solver stores the plan of the current potentials with its rows
// normalised to one, K_ij = exp(x_ij + f_i - log a_i + g_j), and iterates
// scalings u, v over it, f + log u and g + log v being the potentials: two
// FMAs per entry.  When a scaling leaves [2^-300, 2^300] the potentials absorb
// it and K is rebuilt with running maxima.  A column of K may have underflowed
// in part or altogether (g set by rows that are empty, or next to nothing in
// b_j): an entry is off by at most 2^-1075, a column sum by 2^-1075 sum_i a_i
// u_i.  A column sum that is not 2^53 times that is not used: the whole column
// update is then taken with running maxima over the current row potentials,
// and K is rebuilt from its result.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>
#include "dense_common.cuh"
#include "fused.cuh"
#include "fused_ops.cuh"
#include "launch.cuh"

namespace otg {

constexpr int FU_RING = 9;  // most chunks in flight per group
enum { FU_LOG = 0, FU_SCAL = 1, FU_UNB = 2, FU_ABS = 3 };
// Flags that a CTA publishes with its merge.  FU_ABS: FU_BAD_ROW a scaling to
// absorb, FU_BAD_COL a column sum that cannot be used, FU_LOW_COL one that
// cannot if there is a row scaling above 2^30 (FU_LOOSE).
enum { FU_BAD_ROW = 1, FU_BAD_COL = 2, FU_ABORT = 4, FU_LOOSE = 8, FU_LOW_COL = 16 };

template <typename T>
struct FusedArgs {
  const T* M; int64_t ldm; int n, m; T c;
  const T *a, *b, *warm_u, *warm_v;
  int max_iter, period;
  double stop_thr;
  T *u0, *u1, *v0, *v1, *rowc, *fref;   // v0, v1: this CTA's columns of the last two iterates
  unsigned long long *part, *vll, *stll, *ell;   // published words, see Ll
  T* pairs;                  // [grid][m] (maximum, sum) pairs: first and fallback column pass
  T* vfix;                   // [m] v of the fallback column pass
  double* mass;              // [grid] sum of a over the CTA's rows (log forms)
  T *out_u, *out_v;
  double* hist; int hist_cap;
  int* info;                 // status, niter, nchecks, abort
  unsigned* bar;
  uint64_t timeout_ns;
  T fi1, fi2; const T *alw, *bew;
  // split
  int G, kv, mp, mv, gvec, NC;
  int kmat;                  // M holds K = exp(-M/reg) already
  int buf_elems;             // cross-group buffer
};

// ---------------------------------------------------------------------------
// Published values: {value, epoch} in one 64-bit word (float), two such words
// for the halves of a double.  64-bit accesses are single-copy atomic, so a
// word with the expected epoch holds the expected value.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ll_st(unsigned long long* p, unsigned lo, unsigned ep) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" :: "l"(p), "l"(((unsigned long long)ep << 32) | lo) : "memory");
}
__device__ __forceinline__ unsigned long long ll_ld(const unsigned long long* p) {
  unsigned long long x;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
  return x;
}
template <typename T> struct Ll;
template <> struct Ll<float> {
  static constexpr int N = 1;  // words per value
  struct W { unsigned long long w; };
  static __device__ __forceinline__ void put(unsigned long long* p, float x, unsigned ep) { ll_st(p, __float_as_uint(x), ep); }
  static __device__ __forceinline__ W get(const unsigned long long* p) { return W{ll_ld(p)}; }
  static __device__ __forceinline__ bool is(const W& x, unsigned ep) { return (unsigned)(x.w >> 32) == ep; }
  static __device__ __forceinline__ float value(const W& x) { return __uint_as_float((unsigned)x.w); }
};
template <> struct Ll<double> {
  static constexpr int N = 2;
  struct W { unsigned long long a, b; };
  static __device__ __forceinline__ void put(unsigned long long* p, double x, unsigned ep) {
    const unsigned long long e = (unsigned long long)ep << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};"
                 :: "l"(p), "l"(e | (unsigned)__double2loint(x)), "l"(e | (unsigned)__double2hiint(x)) : "memory");
  }
  static __device__ __forceinline__ W get(const unsigned long long* p) {
    W x;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x.a), "=l"(x.b) : "l"(p) : "memory");
    return x;
  }
  static __device__ __forceinline__ bool is(const W& x, unsigned ep) {
    return (unsigned)(x.a >> 32) == ep && (unsigned)(x.b >> 32) == ep;
  }
  static __device__ __forceinline__ double value(const W& x) { return __hiloint2double((int)(unsigned)x.b, (int)(unsigned)x.a); }
};

// Poll one published value (first read `w` done).  Bounded: after timeout_ns,
// or when another thread has given up, raises the abort flag and returns
// false.
template <typename T>
__device__ __forceinline__ bool ll_wait(const unsigned long long* p, unsigned ep, typename Ll<T>::W& w, int* abort_flag,
                                        uint64_t timeout_ns) {
  if (Ll<T>::is(w, ep)) return true;
  unsigned spins = 0;
  uint64_t t0 = 0;
  for (;;) {
    w = Ll<T>::get(p);
    if (Ll<T>::is(w, ep)) return true;
    if ((++spins & 255u) == 0) {
      if (ld_acquire_i(abort_flag)) return false;
      const uint64_t t = globaltimer();
      if (t0 == 0) t0 = t;
      else if (t - t0 > timeout_ns) { atomicExch(abort_flag, 1); return false; }
    }
  }
}

template <typename T>
struct FuSmem { T *vs, *gs, *buf, *data; uint64_t* full; };

// Ring state of a group: the chunk to consume next (slot, parity of its full
// barrier); chunks are numbered on across the passes.
struct FuRing { int slot; uint32_t phase; };

// One vector of the cost from global memory; rows that are not whole 16-byte
// vectors are read element by element, entries beyond the row give `pad`.
template <typename T>
__device__ __forceinline__ void fu_get_global(const FusedArgs<T>& A, int row, int col, T pad, T (&x)[Vec<T>::N]) {
  const T* p = A.M + (int64_t)row * A.ldm + col;
  if (A.gvec) {
    unpack(ld_stream(reinterpret_cast<const typename Vec<T>::type*>(p)), x);
  } else {
#pragma unroll
    for (int w = 0; w < Vec<T>::N; ++w) x[w] = col + w < A.m ? __ldg(p + w) : pad;
  }
}

// A scaling of FU_ABS that needs no absorption: within [2^-300, 2^300].
__device__ __forceinline__ bool fu_tame(double x) { return fu_at_least(x, 0x1p-300) && !fu_at_least(x, 0x1p300); }

// Column sums of the CTA, over the row groups in group order, to its slot.
template <typename T, int NK>
__device__ __forceinline__ void fu_publish_cols(const FusedArgs<T>& A, const FuRow& R, const FuSmem<T>& sm,
                                                const FuV<T> (&acc)[NK], unsigned ep) {
  constexpr int W = Vec<T>::N;
  unsigned long long* dst = A.part + (int64_t)blockIdx.x * A.m * Ll<T>::N;
  if (R.NG == 1) {
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const int col = (k * R.gt + R.tg) * W;
      T x[W];
      acc[k].get(x);
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (col + w < A.m) Ll<T>::put(dst + (col + w) * Ll<T>::N, x[w], ep);
    }
    return;
  }
  if (R.g < R.live) {
    T* b = sm.buf + (int64_t)R.g * A.mp;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      T x[W];
      acc[k].get(x);
      if (k < A.kv) fu_put(b + (k * R.gt + R.tg) * W, x);
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < A.m; j += FU_THREADS) {
    T t = 0;
#pragma unroll 4
    for (int g = 0; g < R.live; ++g) t += sm.buf[g * A.mp + j];
    Ll<T>::put(dst + j * Ll<T>::N, t, ep);
  }
}

// ---------------------------------------------------------------------------
// One pass over the CTA's rows: row updates with sm.vs, scaled entries into
// the CTA's column sums.  q0, q1, q2: scalars of the group's rows, lane l of
// a warp holding row 32 k + l (reloaded every 32 rows unless `held`).
// ---------------------------------------------------------------------------
template <typename T> struct FuHeld {
  T q0, q1, q2;
  // log form (u, log2 a, a): a row of no weight adds nothing to any column
  __device__ __forceinline__ T shift() const { return q2 == T(0) ? T(-INFINITY) : q0 - q1; }
};

template <typename T, int MODE>
__device__ __forceinline__ void fu_fetch(const FusedArgs<T>& A, int row, int end, const T* ucur, FuHeld<T>& H) {
  if (row >= end) return;
  if (MODE == FU_LOG) { H.q0 = __ldcg(ucur + row); H.q1 = A.rowc[row]; H.q2 = A.a[row]; }
  if (MODE == FU_SCAL) H.q1 = A.rowc[row];
  if (MODE == FU_ABS) H.q1 = A.a[row];
  if (MODE == FU_UNB) { H.q0 = __ldcg(ucur + row); H.q1 = A.a[row]; H.q2 = A.alw ? A.alw[row] : T(1); }
}

template <typename T> struct FuTrack { T d0, d1, d2; };

// Row values of a batch from the warps' shares s[]: lane l finishes row
// l / LPR; r is what the row's entries are scaled with in the column sums.
template <typename T, int MODE, int RB, int NK>
__device__ __forceinline__ void fu_rows(const FusedArgs<T>& A, const FuRow& R, T (*red)[FU_WARPS][fu_rb(NK)], T (*rr)[2][fu_rb(NK)],
                                        int& par, T (&s)[RB], int nr, const FuHeld<T>& H, int at, T& t, T& un, T& r, int& flag,
                                        FuTrack<T>& tr) {
  constexpr int LPR = 32 / RB;
  const int myrow = R.lane / LPR, src = at + myrow;
  const T p0 = __shfl_sync(0xffffffffu, H.q0, src), p1 = __shfl_sync(0xffffffffu, H.q1, src),
          p2 = __shfl_sync(0xffffffffu, H.q2, src);
  // FP64 issues at two lanes per clock: the group's first warp alone adds
  // the warps' sums and divides (the log form needs the sum everywhere)
  const bool first_only = sizeof(T) == 8 && MODE != FU_LOG && A.G > 1;
  if (first_only) {
    const T x = fu_scatter<T, RB, false>(s, R.lane);
    if (R.lane % LPR == 0) red[par][R.warp][myrow] = x;
    named_bar(1 + R.g, R.gt);
  } else {
    t = fu_group<T, RB, false>(s, R, A.G, red, par);
  }
  if (!first_only || R.tg < 32) {
    if (first_only) {
      const int l = R.lane % LPR, w0 = R.g * A.G;
      t = 0;
      for (int q = l; q < A.G; q += LPR) t += red[par][w0 + q][myrow];
#pragma unroll
      for (int q = LPR / 2; q > 0; q >>= 1) t += __shfl_xor_sync(0xffffffffu, t, q);
    }
    if (MODE == FU_LOG) {
      // (a row of no weight: its entries are zeros, its sum is not looked at)
      if (p2 == T(0)) t = T(1);
      un = p2 == T(0) ? T(-INFINITY) : p0 - lg2(t);
      r = p2 / t;
    } else if (MODE == FU_SCAL) {
      r = un = T(1) / (p1 * t);
      if (myrow < nr && !isfinite(un)) flag = FU_BAD_ROW;
    } else if (MODE == FU_ABS) {
      un = t;  // (the row's scaling is 1 / t)
      r = p1 / t;
      if (myrow < nr) {
        if (!fu_tame(t)) flag |= FU_BAD_ROW;
        else if (!fu_at_least(t, T(0x1p-30))) flag |= FU_LOOSE;
      }
    } else {
      un = pow_unit(p1 / (p2 * t), A.fi1);
      if (myrow < nr) {
        if (!isfinite(un)) flag = FU_BAD_ROW;
        tr.d0 = pos_max(tr.d0, fabs(un - p0)); tr.d1 = pos_max(tr.d1, fabs(un)); tr.d2 = pos_max(tr.d2, fabs(p0));
      }
      r = p2 * un;
    }
  }
  if (first_only) {
    if (R.tg < 32 && R.lane % LPR == 0) { rr[R.g][0][myrow] = r; rr[R.g][1][myrow] = un; }
    named_bar(1 + R.g, R.gt);
    r = rr[R.g][0][myrow];
    un = rr[R.g][1][myrow];
    par ^= 1;
  }
}

// Running-maximum form of a batch (log form): maxima, then sums of e.
template <typename T, int NK, int RB, typename Arg>
__device__ __forceinline__ void fu_rows_max(const FusedArgs<T>& A, const FuRow& R, T (*red)[FU_WARPS][fu_rb(NK)], int& par, int nr,
                                            FuV<T> (&e)[RB][NK], const FuHeld<T>& H, int at, T& un, T& r, Arg&& arg) {
  constexpr int LPR = 32 / RB;
  T mx[RB], s[RB];
#pragma unroll
  for (int q = 0; q < RB; ++q) mx[q] = -INFINITY;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
#pragma unroll
    for (int q = 0; q < RB; ++q)
      if (q < nr) { e[q][k] = arg(q, k); mx[q] = e[q][k].max_with(mx[q]); }
  }
  const T mg = fu_group<T, RB, true>(mx, R, A.G, red, par);
#pragma unroll
  for (int q = 0; q < RB; ++q) {
    const T m = __shfl_sync(0xffffffffu, mg, q * LPR);
    FuV<T> t = FuV<T>::zero();
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (q < nr) { e[q][k] = FuV<T>::ex_minus(e[q][k], m); t.add_v(e[q][k]); }
    s[q] = t.sum();
  }
  const T t = fu_group<T, RB, false>(s, R, A.G, red, par);
  const int src = at + R.lane / LPR;
  const T p1 = __shfl_sync(0xffffffffu, H.q1, src), p2 = __shfl_sync(0xffffffffu, H.q2, src);
  un = p1 - lse_value(mg, t);
  r = p2 / t;
}

// New row values into memory and into the lane that holds them.
template <typename T, int MODE, int RB>
__device__ __forceinline__ void fu_keep(const FuRow& R, int rb, int at, int nr, T un, T* unxt, FuHeld<T>& H) {
  constexpr int LPR = 32 / RB;
  const int myrow = R.lane / LPR;
  if (R.tg < 32 && R.lane % LPR == 0 && myrow < nr) unxt[rb + myrow] = un;
  if (MODE == FU_LOG || MODE == FU_UNB) {
    const int mine = R.lane - at;
    const T x = __shfl_sync(0xffffffffu, un, (mine >= 0 && mine < RB ? mine : 0) * LPR);
    if (mine >= 0 && mine < nr) H.q0 = x;
  }
}

// RB rows at a time, from shared memory (RES) or the ring.
template <typename T, int MODE, int NK, bool RES>
__device__ __forceinline__ int fu_pass(const FusedArgs<T>& A, const FuRow& R_, const FuSmem<T>& sm,
                                       T (*red)[FU_WARPS][fu_rb(NK)], T (*rr)[2][fu_rb(NK)], FuRing& ring_, const T* ucur, T* unxt,
                                       FuHeld<T>& H_, bool held, FuTrack<T>& tr_, unsigned ep) {
  using V = FuV<T>;
  constexpr int RB = fu_rb(NK), LPR = 32 / RB;
  static_assert(RES || RB == 1, "streamed rows go one at a time");
  // (copies: what the loop reads stays in registers across the inline assembly)
  const FuRow R = R_;
  FuRing ring = ring_;
  FuHeld<T> H = H_;
  FuTrack<T> tr = tr_;
  V acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = V::zero();
  const int kv = A.kv, nc = A.NC, mp = A.mp;
  const uint32_t hop = (uint32_t)R.gt * 16u, pitch = (uint32_t)mp * (uint32_t)sizeof(T);
  const uint32_t va = smem_addr(sm.vs) + (uint32_t)R.tg * 16u;
  const uint32_t chunk = pitch / 2;
  uint32_t xa = smem_addr(sm.data) + (uint32_t)R.tg * 16u;
  if (RES) xa += (uint32_t)(R.ga - R.r0) * pitch;
  else xa += (uint32_t)(R.g * nc) * chunk;
  const typename V::S c = V::all(A.c);
  const bool kmat = A.kmat != 0;
  const int G = A.G, mv = A.mv;
  const T* const Mg = A.M + (int64_t)R.ga * A.ldm;
  const int64_t ldm = A.ldm;
  uint64_t* const full = sm.full + R.g * nc;
  T* const rslot = sm.data + R.g * nc * (mp / 2);
  int par = 0, flag = 0;
  for (int rb = R.ga; rb < R.gb; rb += RB) {
    const int at = (rb - R.ga) & 31;
    if (!held && at == 0) fu_fetch<T, MODE>(A, rb + R.lane, R.gb, ucur, H);
    const int nr = min(RB, R.gb - rb);
    V e[RB][NK];
    T s[RB];
    // The loads and exponentials of a batch stand in one block of code: a
    // branch per vector or row would expose the latency of each (measured
    // 1.4 times slower).  Rows beyond the batch read its last row again;
    // nothing comes of their values.
    auto eval = [&](auto nq) {
#pragma unroll
      for (int q = 0; q < decltype(nq)::value; ++q) {
        const uint32_t xq = xa + min(q, nr - 1) * pitch;
        const typename V::S h = V::all(MODE == FU_LOG ? __shfl_sync(0xffffffffu, H.shift(), at + q) : T(0));
        V t = V::zero();
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const V v = V::lds(va + k * hop), x = V::lds(xq + k * hop);
          if (MODE == FU_LOG) { e[q][k] = V::expo(x, c, v, h); t.add_v(e[q][k]); }
          else { e[q][k] = x; t.fma_v(x, v); }
        }
        s[q] = t.sum();
      }
    };
    if (!RES) {
      // the two halves of the row, each as it lands
      const typename V::S h = V::all(MODE == FU_LOG ? __shfl_sync(0xffffffffu, H.shift(), at) : T(0));
      V t = V::zero();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint32_t xc = xa + (uint32_t)ring.slot * chunk, vc = va + half * (NK / 2) * hop;
        if (!mbar_wait(full + ring.slot, ring.phase, A.info + 3, A.timeout_ns)) flag |= FU_ABORT;
        if (half == 0 || kv > NK / 2) {
#pragma unroll
          for (int kk = 0; kk < NK / 2; ++kk) {
            const int k = half * (NK / 2) + kk;
            const V v = V::lds(vc + kk * hop), x = V::lds(xc + kk * hop);
            if (MODE == FU_LOG) { e[0][k] = V::expo(x, c, v, h); t.add_v(e[0][k]); }
            else { e[0][k] = kmat ? x : V::gibbs(x, c); t.fma_v(e[0][k], v); }
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < NK / 2; ++kk) e[0][half * (NK / 2) + kk] = V::zero();
        }
        if (++ring.slot == nc) { ring.slot = 0; ring.phase ^= 1; }
      }
      s[0] = t.sum();
    } else if (RB > 1 && nr <= RB / 2) {
      eval(std::integral_constant<int, (RB > 1 ? RB / 2 : 1)>{});
#pragma unroll
      for (int q = RB / 2; q < RB; ++q) s[q] = 0;
    } else {
      eval(std::integral_constant<int, RB>{});
    }
    T t, un, r;
    fu_rows<T, MODE, RB, NK>(A, R, red, rr, par, s, nr, H, at, t, un, r, flag, tr);
    if (MODE == FU_LOG) {
      // (the same in every warp of the group)
      if (!__all_sync(0xffffffffu, R.lane / LPR >= nr || fu_near_one(t)))
        fu_rows_max<T, NK, RB>(A, R, red, par, nr, e, H, at, un, r, [&](int q, int k) {
          uint32_t xk = xa + q * pitch + k * hop;
          if (!RES) {
            int sl = ring.slot - (k < NK / 2 ? 2 : 1);  // the row's chunks are still in their slots
            if (sl < 0) sl += nc;
            xk = xa + (uint32_t)sl * chunk + (k % (NK / 2 > 0 ? NK / 2 : 1)) * hop;
          }
          return V::arg(V::lds(xk), c, V::lds(va + k * hop));
        });
    }
    if (!RES && R.tg < 32) {
      // every warp of the group has read the two chunks (the reductions'
      // barriers): their slots take the chunks NC places on
      __syncwarp();
      int s1 = ring.slot - 1;
      if (s1 < 0) s1 += nc;
      const int s0 = s1 == 0 ? nc - 1 : s1 - 1;
      if (R.lane == 0) {
        const int j = 2 * (rb - R.ga) + nc;
        fu_issue(Mg, ldm, mv, mp / 2, R.gb - R.ga, rslot, full, j, s0);
        fu_issue(Mg, ldm, mv, mp / 2, R.gb - R.ga, rslot, full, j + 1, s1);
      }
    }
    fu_keep<T, MODE, RB>(R, rb, at, nr, un, unxt, H);
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      if (q < nr) {
        const typename V::S rq = V::all(__shfl_sync(0xffffffffu, r, q * LPR));
#pragma unroll
        for (int k = 0; k < NK; ++k)
          acc[k].fma_s(e[q][k], rq);
      }
    }
    if (RES) xa += RB * pitch;
  }
  ring_ = ring;
  H_ = H;
  if (MODE == FU_UNB) tr_ = tr;
  fu_publish_cols<T, NK>(A, R, sm, acc, ep);
  return flag;
}

// Absorbing pass of FU_ABS: rows of K with f the exact row update of g = sm.gs
// (running maximum), f into fref, scalings one; K into the resident rows.
template <typename T, int NK>
__device__ __noinline__ void fu_build(const FusedArgs<T>& A, const FuRow& R, const FuSmem<T>& sm, T (*red)[FU_WARPS][fu_rb(NK)],
                                      T* unxt, unsigned ep) {
  constexpr int W = Vec<T>::N;
  const T pad = A.c > T(0) ? T(-INFINITY) : T(INFINITY);
  FuV<T> acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = FuV<T>::zero();
  int par = 0;
  for (int row = R.ga; row < R.gb; ++row) {
    T e[NK][W];
    T one[1] = {T(-INFINITY)};
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const int col = (k * R.gt + R.tg) * W;
      if (k < A.kv) {
        T x[W], v[W];
#pragma unroll
        for (int w = 0; w < W; ++w) x[w] = pad;
        if (col < A.mv) fu_get_global(A, row, col, pad, x);
        fu_get(sm.gs + col, v);
#pragma unroll
        for (int w = 0; w < W; ++w) { e[k][w] = fma(x[w], A.c, v[w]); one[0] = fmax(one[0], e[k][w]); }
      }
    }
    const T mx = fu_group<T, 1, true>(one, R, A.G, red, par);
    one[0] = 0;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      if (k < A.kv) {
#pragma unroll
        for (int w = 0; w < W; ++w) { e[k][w] = ex2(e[k][w] - mx); one[0] += e[k][w]; }
      }
    }
    const T s = fu_group<T, 1, false>(one, R, A.G, red, par);
    const T r = T(1) / s;
    const typename FuV<T>::S ai = FuV<T>::all(A.a[row]);
    T* ks = sm.data + (row - R.r0) * A.mp;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      if (k < A.kv) {
#pragma unroll
        for (int w = 0; w < W; ++w) e[k][w] *= r;
        acc[k].fma_s(FuV<T>::of(e[k]), ai);
        fu_put(ks + (k * R.gt + R.tg) * W, e[k]);
      }
    }
    if (R.tg == 0) {
      A.fref[row] = A.rowc[row] - lse_value(mx, s);
      unxt[row] = T(1);
    }
  }
  fu_publish_cols<T, NK>(A, R, sm, acc, ep);
}

// Column sums alone (scaling forms, first iteration): sum_i K_ij u_i.
template <typename T, int NK, bool RES>
__device__ __noinline__ void fu_colsum(const FusedArgs<T>& A, const FuRow& R, const FuSmem<T>& sm, const T* u, unsigned ep) {
  constexpr int W = Vec<T>::N;
  FuV<T> acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = FuV<T>::zero();
  const T c = A.c;
  for (int row = R.ga; row < R.gb; row += 2) {
    // two rows' loads in flight
    T x[2][NK][W], ui[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = min(row + q, R.gb - 1);
      ui[q] = row + q < R.gb ? __ldcg(u + r) : T(0);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int col = (k * R.gt + R.tg) * W;
        if (RES) { if (k < A.kv) fu_get(sm.data + (r - R.r0) * A.mp + col, x[q][k]); }
        else fu_get_global(A, r, col < A.mv ? col : 0, T(0), x[q][k]);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int k = 0; k < NK; ++k)
        if (!RES || k < A.kv) {
          const FuV<T> xv = FuV<T>::of(x[q][k]);
          acc[k].fma_s(RES || A.kmat ? xv : FuV<T>::gibbs(xv, FuV<T>::all(c)), FuV<T>::all(ui[q]));
        }
  }
  fu_publish_cols<T, NK>(A, R, sm, acc, ep);
}

// Column log-sum-exps alone (log forms: first iteration and the fallback):
// (maximum, sum) pairs of x_ij + u_i over the CTA's rows, sixteen loads of a
// thread in flight: four rows of four vectors.  MARKED: only vectors with a
// column whose sm.vs is NaN, sixteen rows of one, as few threads have several
// (8192^2 float32, an eighth of the columns marked: four by four 67 us).
template <typename T, bool TILE, bool MARKED>
__device__ __noinline__ void fu_collse(const FusedArgs<T>& A_, const FuRow& R_, const FuSmem<T>& sm_, const T* u) {
  constexpr int W = Vec<T>::N, KB = MARKED ? 1 : 4, RW = 16 / KB;
  const FusedArgs<T> A = A_;
  const FuRow R = R_;
  const FuSmem<T> sm = sm_;
  const T pad = A.c > T(0) ? T(-INFINITY) : T(INFINITY);
  for (int k0 = 0; k0 < A.kv; k0 += KB) {
    T mx[KB][W], s[KB][W];
#pragma unroll
    for (int k = 0; k < KB; ++k)
#pragma unroll
      for (int w = 0; w < W; ++w) { mx[k][w] = -INFINITY; s[k][w] = 0; }
    bool on = true;
    if (MARKED) {
      const int at = (k0 * R.gt + R.tg) * W;
      T v[W];
      fu_get(sm.vs + at, v);
      on = false;
#pragma unroll
      for (int w = 0; w < W; ++w) on |= at + w < A.m && isnan(v[w]);
      if (!__syncthreads_or(on)) continue;
    }
    // one rescaling exponential per column for the rows of an update
    for (int row = on ? R.ga : R.gb; row < R.gb; row += RW) {
      T ui[RW];
#pragma unroll
      for (int q = 0; q < RW; ++q) ui[q] = row + q < R.gb ? __ldcg(u + row + q) : T(-INFINITY);
      // (vectors beyond the row read its first one and are not stored)
      T x[KB][RW][W];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int at = ((k0 + k) * R.gt + R.tg) * W, col = at < A.mv ? at : 0;
#pragma unroll
        for (int q = 0; q < RW; ++q) {
          const int r = min(row + q, R.gb - 1);
          if (TILE) fu_get(sm.data + (r - R.r0) * A.mp + col, x[k][q]);
          else if (MARKED) unpack(ld_stream(reinterpret_cast<const typename Vec<T>::type*>(A.M + (int64_t)r * A.ldm + col)), x[k][q]);
          else fu_get_global(A, r, col, pad, x[k][q]);
        }
      }
#pragma unroll
      for (int k = 0; k < KB; ++k) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
          T t[RW], top = mx[k][w];
#pragma unroll
          for (int q = 0; q < RW; ++q) { t[q] = row + q < R.gb ? fma(x[k][q][w], A.c, ui[q]) : T(-INFINITY); top = fmax(top, t[q]); }
          // (an empty column so far: the sums stay zero)
          const T ref = top == -INFINITY ? T(0) : top;
          T sum = s[k][w] * ex2(mx[k][w] - ref);
#pragma unroll
          for (int q = 0; q < RW; ++q) sum += ex2(t[q] - ref);
          s[k][w] = sum;
          mx[k][w] = top;
        }
      }
    }
    // over the row groups: the largest maximum first, then the rescaled sums
    // (a group without rows brings empty pairs)
    if (R.NG > 1) {
      T* b = sm.buf + R.g * A.mp;
#pragma unroll
      for (int k = 0; k < KB; ++k)
        if (k0 + k < A.kv) fu_put(b + ((k0 + k) * R.gt + R.tg) * W, mx[k]);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int col = ((k0 + k) * R.gt + R.tg) * W;
        if (k0 + k < A.kv) {
#pragma unroll
          for (int w = 0; w < W; ++w) {
            T top = -INFINITY;
            for (int g = 0; g < R.NG; ++g) top = fmax(top, sm.buf[g * A.mp + col + w]);
            if (top != -INFINITY) s[k][w] *= ex2(mx[k][w] - top);
            mx[k][w] = top;
          }
        }
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < KB; ++k)
        if (k0 + k < A.kv) fu_put(b + ((k0 + k) * R.gt + R.tg) * W, s[k]);
      __syncthreads();
    }
    if (R.g == 0) {
      T* dst = A.pairs + 2 * (int64_t)blockIdx.x * A.m;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int col = ((k0 + k) * R.gt + R.tg) * W;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          if (k0 + k < A.kv && col + w < A.m) {
            T t = s[k][w];
            if (R.NG > 1) {
              t = 0;
              for (int g = 0; g < R.NG; ++g) t += sm.buf[g * A.mp + col + w];
            }
            dst[2 * (col + w)] = mx[k][w];
            dst[2 * (col + w) + 1] = t;
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Merge: this CTA's share of the columns over the grid's slots.  LC lanes
// take adjacent columns and 32 / LC lanes share a column's slots, as do `per`
// warps; partial sums are added in lane and warp order, so the sum of a
// column is the same in every run.  fin(j, s) finishes column j.
// ---------------------------------------------------------------------------
template <typename T, typename Fin>
__device__ __forceinline__ bool fu_merge(const FusedArgs<T>& A, const FuRow& R, T* s_s, unsigned ep, Fin&& fin) {
  const int np = gridDim.x;
  const int cb = (int)((int64_t)A.m * blockIdx.x / gridDim.x), ce = (int)((int64_t)A.m * (blockIdx.x + 1) / gridDim.x);
  const int mc = ce - cb;
  int LC = 32;
  while (LC > 4 && LC / 2 >= mc) LC /= 2;
  const int SL = 32 / LC, ncb = (mc + LC - 1) / LC;
  const int per = ncb >= FU_WARPS ? 1 : (ncb ? FU_WARPS / ncb : 1);
  const int at_once = FU_WARPS / per;
  const int sub = R.warp % per, mine = R.warp / per;
  const int step = per * SL;
  bool ok = true;
  if (mc == 0) {
    // (a grid of more than m CTAs; a slot is not rewritten before this CTA's flags are out)
    for (int p = threadIdx.x; p < np && ok; p += FU_THREADS) {
      const unsigned long long* q = A.part + (int64_t)p * A.m * Ll<T>::N;
      typename Ll<T>::W x = Ll<T>::get(q);
      ok = ll_wait<T>(q, ep, x, A.info + 3, A.timeout_ns);
    }
    return __syncthreads_and(ok);
  }
  for (int b0 = 0; b0 < ncb; b0 += at_once) {
    const int blk = b0 + mine;
    const int j = cb + blk * LC + R.lane % LC;
    const bool live = mine < at_once && blk < ncb && j < ce;
    T s = 0;
    if (live) {
      constexpr int U = sizeof(T) == 8 ? 4 : 8;
      const int64_t stride = (int64_t)step * A.m * Ll<T>::N;
      int p = sub * SL + R.lane / LC;
      const unsigned long long* q = A.part + ((int64_t)p * A.m + j) * Ll<T>::N;
      for (; p < np; p += U * step, q += U * stride) {
        typename Ll<T>::W x[U];
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (p + k * step < np) x[k] = Ll<T>::get(q + k * stride);
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (p + k * step < np) {
            ok = ok && ll_wait<T>(q + k * stride, ep, x[k], A.info + 3, A.timeout_ns);
            s += Ll<T>::value(x[k]);
          }
      }
    }
    __syncwarp();
    for (int o = LC; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (per > 1) {
      s_s[R.warp * 32 + R.lane] = s;
      __syncthreads();
      if (live && sub == 0 && R.lane < LC)
        for (int q = 1; q < per; ++q) s += s_s[(R.warp + q) * 32 + R.lane];
      __syncthreads();
    }
    if (live && sub == 0 && R.lane < LC) fin(j, s);
  }
  return ok;
}

// The same of (maximum, sum) pairs, behind a grid barrier: the column update
// log2 b - log2 sum exp into vfix and, as epoch `pub`, the published v.  `ep`:
// only columns whose v of that epoch is NaN.  Blocks of 32 columns go around
// the CTAs (the marked ones are neighbours), a block's slots around the warps.
// Out of line: it runs once or for columns that underflowed, and its registers
// must not weigh on the passes.
template <typename T>
__device__ __noinline__ void fu_merge_pairs(const FusedArgs<T>& A, T* s_s, T* s_m, unsigned ep, unsigned pub) {
  constexpr int U = 10;  // slots of a warp in flight (19 of 152)
  const int warp = threadIdx.x >> 5, np = gridDim.x;
  for (int j0 = 32 * blockIdx.x; j0 < A.m; j0 += 32 * gridDim.x) {
    const int j = j0 + (threadIdx.x & 31);
    bool live = j < A.m;
    if (ep) {
      if (live) live = isnan(Ll<T>::value(Ll<T>::get(A.vll + j * Ll<T>::N)));
      if (!__any_sync(0xffffffffu, live)) continue;  // (the same in every warp)
    }
    T mx = -INFINITY, s = 0;
    if (live)
      for (int p = warp; p < np; p += U * FU_WARPS) {
        T m2[U], s2[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const bool in = p + k * FU_WARPS < np;
          const T* q = A.pairs + 2 * ((int64_t)(in ? p + k * FU_WARPS : p) * A.m + j);
          m2[k] = in ? __ldcg(q) : T(-INFINITY);
          s2[k] = in ? __ldcg(q + 1) : T(0);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) lse_merge(mx, s, m2[k], s2[k]);
      }
    s_s[threadIdx.x] = s;
    s_m[threadIdx.x] = mx;
    __syncthreads();
    if (live && warp == 0) {
      for (int q = 1; q < FU_WARPS; ++q) lse_merge(mx, s, s_m[q * 32 + threadIdx.x], s_s[q * 32 + threadIdx.x]);
      const T vn = lg2(A.b[j]) - lse_value(mx, s);
      A.vfix[j] = vn;
      if (pub) Ll<T>::put(A.vll + j * Ll<T>::N, vn, pub);
    }
    __syncthreads();
  }
}

// The flags that any thread of the CTA has.
__device__ __forceinline__ int fu_any(int bits) {
  int all = 0;
  if (__syncthreads_or(bits))
    for (int f = 1; f <= FU_LOW_COL; f <<= 1)
      if (__syncthreads_or(bits & f)) all |= f;
  return all;
}

// The whole v of epoch `ep` into sm.vs (poll), the flags that the CTAs
// published with it, and with `check` their error shares added in CTA order.
// Every thread gets the same flags and error.
template <typename T>
__device__ __forceinline__ int fu_collect(const FusedArgs<T>& A, const FuSmem<T>& sm, unsigned ep, bool check, bool ok,
                                          double& e2) {
  int bits = ok ? 0 : FU_ABORT;
  constexpr int U = 4;
  for (int j = threadIdx.x; j < A.m; j += U * FU_THREADS) {
    typename Ll<T>::W x[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (j + k * FU_THREADS < A.m) x[k] = Ll<T>::get(A.vll + (j + k * FU_THREADS) * Ll<T>::N);
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (j + k * FU_THREADS < A.m) {
        if (!bits && !ll_wait<T>(A.vll + (j + k * FU_THREADS) * Ll<T>::N, ep, x[k], A.info + 3, A.timeout_ns)) bits = FU_ABORT;
        sm.vs[j + k * FU_THREADS] = Ll<T>::value(x[k]);
      }
  }
  double share = 0.0;
  for (int p = threadIdx.x; p < (int)gridDim.x; p += FU_THREADS) {
    Ll<float>::W st = Ll<float>::get(A.stll + p);
    if (!(bits & FU_ABORT) && !ll_wait<float>(A.stll + p, ep, st, A.info + 3, A.timeout_ns)) bits = FU_ABORT;
    if (!(bits & FU_ABORT)) bits |= (int)(unsigned)st.w;
    if (check) {
      Ll<double>::W w = Ll<double>::get(A.ell + 2 * p);
      if (!(bits & FU_ABORT) && !ll_wait<double>(A.ell + 2 * p, ep, w, A.info + 3, A.timeout_ns)) bits |= FU_ABORT;
      share += Ll<double>::value(w);
    }
  }
  const int all = fu_any(bits);
  if (check) e2 = block_sum_fixed(share);
  return all;
}

template <typename T, int MODE, int NK, bool RES>
__global__ void __launch_bounds__(FU_THREADS, 1) fused_sinkhorn_kernel(const __grid_constant__ FusedArgs<T> A) {
  extern __shared__ __align__(16) unsigned char fu_smem[];
  __shared__ T red[2][FU_WARPS][fu_rb(NK)];
  __shared__ T rr[FU_WARPS][2][fu_rb(NK)];
  __shared__ T s_s[FU_WARPS * 32];
  constexpr int W = Vec<T>::N;
  constexpr bool LOGF = MODE == FU_LOG || MODE == FU_ABS;
  FuRow R;
  R.r0 = (int)((int64_t)A.n * blockIdx.x / gridDim.x);
  R.r1 = (int)((int64_t)A.n * (blockIdx.x + 1) / gridDim.x);
  R.warp = threadIdx.x >> 5;
  R.lane = threadIdx.x & 31;
  R.NG = FU_WARPS / A.G;
  R.g = R.warp / A.G;
  R.gt = A.G * 32;
  R.tg = threadIdx.x - R.g * R.gt;
  {
    // rows per group; float64: whole batches, as a reduction costs the same
    // FP64 operations for one row as for a batch
    constexpr int RB = fu_rb(NK);
    const int rows = R.r1 - R.r0;
    int per = (rows + R.NG - 1) / R.NG;
    if (sizeof(T) == 8) per = (per + RB - 1) / RB * RB;
    R.live = (rows + per - 1) / per;
    R.ga = min(R.r1, R.r0 + per * R.g);
    R.gb = min(R.r1, R.ga + per);
  }
  FuSmem<T> sm;
  sm.vs = reinterpret_cast<T*>(fu_smem);
  sm.gs = sm.vs + (MODE == FU_ABS ? A.mp : 0);
  sm.buf = sm.gs + A.mp;
  sm.full = reinterpret_cast<uint64_t*>(sm.buf + A.buf_elems);  // streamed: NG x NC barriers
  sm.data = reinterpret_cast<T*>(sm.full + (RES ? 0 : (R.NG * A.NC + 1) / 2 * 2));
  T* s_m = R.NG > 1 ? sm.buf : sm.vs;  // maxima of the pairs merge (free then: the next v overwrites vs)
  int* abort_flag = A.info + 3;
  unsigned gen = 0;
  const T L2E = T(OTG_LOG2E), LN2 = T(OTG_LN2);
  const int cb = (int)((int64_t)A.m * blockIdx.x / gridDim.x), ce = (int)((int64_t)A.m * (blockIdx.x + 1) / gridDim.x);

  // initial state: this CTA's rows, its share of the columns, its published words
  for (int i = R.r0 + threadIdx.x; i < R.r1; i += FU_THREADS) {
    if (MODE == FU_LOG) { A.u0[i] = A.warm_u ? A.warm_u[i] * L2E : T(0); A.rowc[i] = lg2(A.a[i]); }
    if (MODE == FU_ABS) { A.fref[i] = A.warm_u ? A.warm_u[i] * L2E : T(0); A.u0[i] = T(1); A.rowc[i] = lg2(A.a[i]); }
    if (MODE == FU_SCAL) { A.u0[i] = A.warm_u ? exp(A.warm_u[i]) : T(1) / T(A.n); A.rowc[i] = T(1) / A.a[i]; }
    if (MODE == FU_UNB) A.u0[i] = A.warm_u ? exp(A.warm_u[i]) : T(1);
  }
  for (int j = cb + threadIdx.x; j < ce; j += FU_THREADS) {
    // iteration -1: what a solve that stops before its first iterate returns
    if (LOGF) A.v1[j] = A.warm_v ? A.warm_v[j] * L2E : T(0);
    if (MODE == FU_SCAL) A.v1[j] = A.warm_v ? exp(A.warm_v[j]) : T(1) / T(A.m);
    if (MODE == FU_UNB) A.v1[j] = A.warm_v ? exp(A.warm_v[j]) : T(1);
    for (int w = 0; w < Ll<T>::N; ++w) A.vll[j * Ll<T>::N + w] = 0ull;
  }
  for (int j = threadIdx.x; j < A.m * Ll<T>::N; j += FU_THREADS) A.part[(int64_t)blockIdx.x * A.m * Ll<T>::N + j] = 0ull;
  if (LOGF) {
    double w = 0.0;
    for (int i = R.r0 + threadIdx.x; i < R.r1; i += FU_THREADS) w += widen(A.a[i]);
    w = block_sum_fixed(w);
    if (threadIdx.x == 0) A.mass[blockIdx.x] = w;
  }
  if (threadIdx.x < 12) A.ell[(int64_t)12 * blockIdx.x + threadIdx.x] = 0ull;
  if (threadIdx.x == 0) A.stll[blockIdx.x] = 0ull;
  // beyond the row: v that adds nothing
  const T vpad = MODE == FU_LOG ? T(-INFINITY) : T(0);
  for (int j = threadIdx.x; j < A.mp; j += FU_THREADS) { if (MODE == FU_ABS) sm.gs[j] = 0; sm.vs[j] = vpad; }
  // resident rows: every thread loads the vectors that it will read
  if (RES && MODE != FU_ABS) {
    const T pad = MODE != FU_LOG ? T(0) : (A.c > T(0) ? T(-INFINITY) : T(INFINITY));
    for (int row = R.ga; row < R.gb; ++row) {
      T* dst = sm.data + (row - R.r0) * A.mp;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int col = (k * R.gt + R.tg) * W;
        if (k < A.kv) {
          T x[W];
#pragma unroll
          for (int w = 0; w < W; ++w) x[w] = pad;
          if (col < A.mv) fu_get_global(A, row, col, pad, x);
          if (MODE != FU_LOG && !A.kmat) {
#pragma unroll
            for (int w = 0; w < W; ++w) x[w] = col + w < A.m ? ex2(x[w] * A.c) : T(0);
          }
          fu_put(dst + col, x);
        }
      }
    }
  }
  // the ring: zeros beyond the rows (the copies never write there)
  FuRing ring{0, 0u};
  if (!RES) {
    const int chunk = A.mp / 2;
    for (int j = threadIdx.x; j < R.NG * A.NC * chunk; j += FU_THREADS) sm.data[j] = T(0);
    for (int j = threadIdx.x; j < R.NG * A.NC; j += FU_THREADS) mbar_init(sm.full + j, 1);
    fence_mbar_init();
    fence_proxy_async_smem();
    __syncthreads();
    if (R.tg == 0 && R.gb > R.ga)
      for (int q = 0; q < A.NC; ++q)
        fu_issue(A.M + (int64_t)R.ga * A.ldm, A.ldm, A.mv, A.mp / 2, R.gb - R.ga, sm.data + R.g * A.NC * (A.mp / 2),
                 sm.full + R.g * A.NC, q, q);
  }
  bool ok = fu_barrier(A.bar, gen, abort_flag, A.timeout_ns);  // the published words are cleared everywhere

  // u, v of the last two iterates (v: this CTA's columns): ucur, vcur are
  // iteration ii - 1 at the head of the loop
  T *ucur = A.u0, *unxt = A.u1;
  T *vcur = A.v1, *vnxt = A.v0;
  int nchk = 0, status = OTG_STATUS_MAXITER, niter = A.max_iter - 1;
  double e2 = 0.0;
  FuHeld<T> H{T(0), T(0), T(0)};
  const bool held = R.gb - R.ga <= 32;
  if (held) fu_fetch<T, MODE>(A, R.ga + R.lane, R.gb, ucur, H);

  if (MODE == FU_UNB) {
    for (int j = threadIdx.x; j < A.m; j += FU_THREADS)
      sm.vs[j] = (A.bew ? A.bew[j] : T(1)) * (A.warm_v ? exp(A.warm_v[j]) : T(1));
    __syncthreads();
    __shared__ T s_mx[6][FU_WARPS];
    for (int ii = 0; ok && ii < A.max_iter; ++ii) {
      const unsigned ep = (unsigned)ii + 2u;
      FuTrack<T> ut{T(-INFINITY), T(-INFINITY), T(-INFINITY)}, vt = ut;
      int flag = fu_pass<T, MODE, NK, RES>(A, R, sm, red, rr, ring, ucur, unxt, H, held, ut, ep);
      ok = fu_merge<T>(A, R, s_s, ep, [&](int j, T s) {
        const T be = A.bew ? A.bew[j] : T(1);
        const T vn = pow_unit(A.b[j] / (be * s), A.fi2);
        if (s == T(0) || !isfinite(vn)) flag |= FU_BAD_COL;
        const T vo = __ldcg(vcur + j);
        vnxt[j] = vn;
        Ll<T>::put(A.vll + j * Ll<T>::N, be * vn, ep);
        vt.d0 = pos_max(vt.d0, fabs(vn - vo));
        vt.d1 = pos_max(vt.d1, fabs(vn));
        vt.d2 = pos_max(vt.d2, fabs(vo));
      });
      // this CTA's maxima and flags
      T mine[6] = {ut.d0, ut.d1, ut.d2, vt.d0, vt.d1, vt.d2};
#pragma unroll
      for (int q = 0; q < 6; ++q) { mine[q] = warp_pos_max(mine[q]); if (R.lane == 0) s_mx[q][R.warp] = mine[q]; }
      if (flag & FU_ABORT) ok = false;
      flag = __syncthreads_or(flag);  // either flag ends the solve with the previous pair
      if (threadIdx.x < 6) {
        T t = s_mx[threadIdx.x][0];
        for (int w = 1; w < FU_WARPS; ++w) t = pos_max(t, s_mx[threadIdx.x][w]);
        Ll<T>::put(A.ell + 12 * (int64_t)blockIdx.x + 2 * threadIdx.x, t, ep);
      }
      if (threadIdx.x == 0) ll_st(A.stll + blockIdx.x, flag ? FU_BAD_ROW : 0, ep);
      const int got = fu_collect(A, sm, ep, false, ok, e2);
      if (got & FU_ABORT) { ok = false; break; }
      // everyone's maxima, all six words in flight at once; one warp alone
      // does the FP64 of the error (2000 x 3000 float32: 14.9 us per iteration
      // with a trip to L2 per word and eight warps' conversions, now 14.1)
      T mx[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) mx[q] = -INFINITY;
      for (int p = threadIdx.x; p < (int)gridDim.x; p += FU_THREADS) {
        const unsigned long long* w = A.ell + 12 * (int64_t)p;
        typename Ll<T>::W x[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) x[q] = Ll<T>::get(w + 2 * q);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          ok = ok && ll_wait<T>(w + 2 * q, ep, x[q], A.info + 3, A.timeout_ns);
          mx[q] = pos_max(mx[q], Ll<T>::value(x[q]));
        }
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) { mx[q] = warp_pos_max(mx[q]); if (R.lane == 0) s_mx[q][R.warp] = mx[q]; }
      if (__syncthreads_or(!ok)) { ok = false; break; }
      int stop = 0;
      if (threadIdx.x == 0) {
        double mk[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          T t = s_mx[q][0];
          for (int w = 1; w < FU_WARPS; ++w) t = pos_max(t, s_mx[q][w]);
          mk[q] = widen(t);
        }
        const double err = 0.5 * (mk[0] / fmax(fmax(mk[1], mk[2]), 1.0) + mk[3] / fmax(fmax(mk[4], mk[5]), 1.0));
        if (blockIdx.x == 0 && ii < A.hist_cap && !(got & FU_BAD_ROW)) A.hist[ii] = err;
        stop = err < A.stop_thr;
      }
      stop = __syncthreads_or(stop);
      if (got & FU_BAD_ROW) { status = OTG_STATUS_NUMERICAL; niter = ii; break; }  // previous pair kept
      nchk = ii + 1;
      T* t;
      t = ucur; ucur = unxt; unxt = t;
      t = vcur; vcur = vnxt; vnxt = t;
      if (stop) { status = OTG_STATUS_CONVERGED; niter = ii; break; }
    }
  } else if (ok && A.max_iter > 0) {
    // column update of the initial row potentials: the first v (FU_ABS takes
    // it when it builds K)
    int flag = 0, got = 0;
    if (MODE != FU_ABS) {
      if (LOGF) {
        fu_collse<T, RES, false>(A, R, sm, ucur);
        ok = fu_barrier(A.bar, gen, abort_flag, A.timeout_ns);
        if (ok) fu_merge_pairs(A, s_s, s_m, 0u, 1u);
      } else {
        fu_colsum<T, NK, RES>(A, R, sm, ucur, 1u);
        ok = fu_merge<T>(A, R, s_s, 1u, [&](int j, T s) {
          const T vn = A.b[j] / s;
          if (s == T(0) || !isfinite(vn)) flag |= FU_BAD_COL;
          Ll<T>::put(A.vll + j * Ll<T>::N, vn, 1u);
        });
      }
      flag = __syncthreads_or(flag) ? FU_BAD_COL : 0;
      if (threadIdx.x == 0) ll_st(A.stll + blockIdx.x, flag, 1u);
      got = fu_collect(A, sm, 1u, false, ok, e2);
      if (got & FU_ABORT) ok = false;
    }
    // FU_ABS: K is to be built, from a column update of its own (else the
    // scalings are absorbed)
    bool build = MODE == FU_ABS, absolute = true;
    // Column sums below s_lim[1] may have lost bits to underflow (FU_ABS: with
    // row scalings up to 2^300, s_lim[0] up to 2^30): a part of the mass, and
    // no less than the roundings of denormals.
    __shared__ T s_lim[2];  // (registers are what the passes have least of)
    if (LOGF) {
      double w = 0.0;
      for (int p = threadIdx.x; p < (int)gridDim.x; p += FU_THREADS) w += __ldcg(A.mass + p);
      w = block_sum_fixed(w);
      if (threadIdx.x == 0) {
        s_lim[0] = (T)fmax(w * 0x1p-992, 0x1p-1000);
        s_lim[1] = (T)(MODE == FU_ABS ? fmax(w * 0x1p-722, 0x1p-1000) : sizeof(T) == 8 ? fmax(w * 0x1p-985, 0x1p-1000)
                                                                                       : fmax(w * 0x1p-70, 0x1p-100));
      }
    }
    for (int ii = 0; ok; ++ii) {
      // sm.vs holds v of iteration ii, ucur u of iteration ii - 1
      if (MODE == FU_SCAL && (got & FU_BAD_COL)) {
        // zero column sum or non-finite v: the previous pair
        status = OTG_STATUS_NUMERICAL; niter = ii; break;
      }
      const unsigned ep = (unsigned)ii + 2u;
      FuTrack<T> tr{T(0), T(0), T(0)};
      flag = 0;
      if (MODE == FU_ABS && build) {
        if (absolute) {
          // the first column update, or a column sum that cannot be used:
          // the update of the current row potentials, with running maxima
          for (int i = R.r0 + threadIdx.x; i < R.r1; i += FU_THREADS) A.fref[i] = __ldcg(A.fref + i) - lg2(__ldcg(ucur + i));
          __syncthreads();
          fu_collse<T, false, false>(A, R, sm, A.fref);
          if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
          fu_merge_pairs(A, s_s, s_m, 0u, 0u);
          if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        }
        for (int j = threadIdx.x; j < A.mp; j += FU_THREADS) {
          if (j < A.m) sm.gs[j] = absolute ? __ldcg(A.vfix + j) : sm.gs[j] + lg2(sm.vs[j]);
          sm.vs[j] = j < A.m ? T(1) : T(0);
        }
        absolute = false;
        __syncthreads();
        fu_build<T, NK>(A, R, sm, red, unxt, ep);
      } else {
        flag = fu_pass<T, MODE, NK, RES>(A, R, sm, red, rr, ring, ucur, unxt, H, held, tr, ep);
      }
      T* t;
      t = ucur; ucur = unxt; unxt = t;
      t = vcur; vcur = vnxt; vnxt = t;
      const bool check = ii % A.period == 0, last = ii + 1 == A.max_iter;
      e2 = 0.0;
      ok = fu_merge<T>(A, R, s_s, ep, [&](int j, T s) {
        const T bj = A.b[j], vo = sm.vs[j];
        vcur[j] = vo;
        if (check) {
          // column marginal of (u, v) of iteration ii
          const double d = widen(MODE == FU_LOG ? s : vo * s) - widen(bj);
          e2 += d * d;
        }
        T vn;
        if (MODE == FU_LOG) {
          vn = bj == T(0) ? T(-INFINITY) : vo + lg2(bj / s);
          if (bj != T(0) && !fu_at_least(s, s_lim[1])) { flag |= FU_BAD_COL; vn = T(NAN); }
        } else if (MODE == FU_ABS) {
          vn = bj == T(0) ? T(1) : bj / s;
          if (bj != T(0)) {
            if (!fu_at_least(s, s_lim[1])) flag |= fu_at_least(s, s_lim[0]) ? FU_LOW_COL : FU_BAD_COL;
            if (!fu_tame(vn)) flag |= fu_at_least(vn, T(0x1p-900)) ? FU_BAD_ROW : FU_BAD_COL;  // (a denormal quotient)
          }
        } else {
          vn = bj / s;
          if (s == T(0) || !isfinite(vn)) flag |= FU_BAD_COL;
        }
        Ll<T>::put(A.vll + j * Ll<T>::N, vn, ep);
      });
      if (check) {
        e2 = block_sum_fixed(e2);
        if (threadIdx.x == 0) Ll<double>::put(A.ell + 2 * blockIdx.x, e2, ep);
      }
      if (flag & FU_ABORT) ok = false;
      const int mine = fu_any(flag & ~FU_ABORT);
      if (threadIdx.x == 0) ll_st(A.stll + blockIdx.x, mine, ep);
      got = fu_collect(A, sm, ep, check, ok, e2);
      if (got & FU_ABORT) { ok = false; break; }
      if (MODE == FU_SCAL && (got & FU_BAD_ROW)) {
        // non-finite u: the previous pair
        t = ucur; ucur = unxt; unxt = t;
        t = vcur; vcur = vnxt; vnxt = t;
        status = OTG_STATUS_NUMERICAL; niter = ii; break;
      }
      if (check) {
        if (blockIdx.x == 0 && threadIdx.x == 0) A.hist[nchk < A.hist_cap ? nchk : A.hist_cap - 1] = e2;
        ++nchk;
        // (one warp's square root: FP64 issues at two lanes per clock)
        if (__syncthreads_or(threadIdx.x == 0 && sqrt(e2) < A.stop_thr)) { status = OTG_STATUS_CONVERGED; niter = ii; break; }
      }
      if (last) { niter = ii; break; }
      if (MODE == FU_ABS) {
        absolute = (got & FU_BAD_COL) || ((got & FU_LOW_COL) && (got & FU_LOOSE));
        build = absolute || (got & FU_BAD_ROW);
      }
      if (MODE == FU_LOG && (got & FU_BAD_COL)) {
        // column sums too small to trust (NaN in v): their update with running maxima
        fu_collse<T, RES, true>(A, R, sm, ucur);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        fu_merge_pairs(A, s_s, s_m, ep, 0u);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        for (int j = threadIdx.x; j < A.m; j += FU_THREADS) {  // (sm.vs was the merge's scratch)
          const T v = Ll<T>::value(Ll<T>::get(A.vll + j * Ll<T>::N));
          sm.vs[j] = isnan(v) ? __ldcg(A.vfix + j) : v;
        }
        __syncthreads();
      }
    }
  }
  if (!RES) {
    // copies in flight land before the CTA leaves: NC chunks from the one due next
    const uint64_t t0 = globaltimer();
    if (R.tg == 0 && R.gb > R.ga)
      for (int q = 0; q < A.NC; ++q) {
        while (!mbar_try_wait(sm.full + R.g * A.NC + ring.slot, ring.phase)) if (globaltimer() - t0 > A.timeout_ns) break;
        if (++ring.slot == A.NC) { ring.slot = 0; ring.phase ^= 1; }
      }
  }
  __syncthreads();
  if (!ok) return;

  // Final state in natural units: this CTA's rows and its share of the columns.
  for (int i = R.r0 + threadIdx.x; i < R.r1; i += FU_THREADS) {
    const T u = __ldcg(ucur + i);
    A.out_u[i] = MODE == FU_LOG ? u * LN2 : MODE == FU_ABS ? (__ldcg(A.fref + i) - lg2(u)) * LN2 : u;
  }
  for (int j = cb + threadIdx.x; j < ce; j += FU_THREADS) {
    const T v = __ldcg(vcur + j);
    // FU_ABS: scalings over the absorbed potentials (none yet when max_iter is 0)
    A.out_v[j] = MODE == FU_LOG ? v * LN2 : MODE == FU_ABS ? (A.max_iter > 0 ? sm.gs[j] + lg2(v) : v) * LN2 : v;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.info[0] = status;
    A.info[1] = niter;
    A.info[2] = nchk;
  }
}

// ---------------------------------------------------------------------------
// Streamed rows that are not whole 16-byte vectors: one copy into padded rows
// (scaling forms: of K = exp(-M/reg), unless that is what M holds already).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) fused_pack_kernel(const T* __restrict__ M, int64_t n, int64_t m, int64_t ldm, T c,
                                                         int expo, T pad, T* __restrict__ out, int64_t ldo) {
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x)
    for (int j = threadIdx.x; j < ldo; j += blockDim.x) {
      const T x = j < m ? M[i * ldm + j] : pad;
      out[i * ldo + j] = expo && j < m ? ex2(x * c) : x;
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct FuPlan { int grid, G, NK, kv, mp, res, NC, buf_elems; size_t smem; };

// The kernels' static shared memory (merge and reduction scratch), rounded up.
template <typename T> size_t fu_static_smem(int nk) {
  return sizeof(T) * (FU_WARPS * (32 + 6 + 4 * (size_t)fu_rb(nk))) + 304;
}

struct FuDevice { int sms = 0; size_t smem = 0; };
inline FuDevice fu_device() {
  FuDevice d;
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  d.smem = v > 0 ? (size_t)v : 0;
  return d;
}

// CTAs: one per SM at most, each with a row.  Small problems take fewer, and
// a share of a few rows is rounded up to whole batches, as a CTA's time is
// that of its batches (n = m = 1024: 128 CTAs of 8 rows 5.5 us per iteration
// in float32 and 10.8 in float64, 152 CTAs of 7 rows 6.4 and 11.2).
template <typename T>
int fu_grid(int64_t n, int64_t m, int requested, int sms) {
  const int64_t least = sizeof(T) == 4 ? 4096 : 1024;  // entries per CTA
  int64_t g = (n * m + least - 1) / least;
  g = std::max<int64_t>(std::min<int64_t>(std::min<int64_t>(g, sms), n), 1);
  const int64_t V = (m + Vec<T>::N - 1) / Vec<T>::N;
  int nk = 1;
  while (nk < 16 && (int64_t)FU_WARPS * 32 * nk < V) nk *= 2;
  const int64_t rb = fu_rb(nk), rows = (n + g - 1) / g;
  if (rows < 2 * rb) {
    const int64_t up = (rows + rb - 1) / rb * rb;
    g = (n + up - 1) / up;
  }
  if (requested > 0) g = std::min<int64_t>(g, requested);
  return (int)g;
}

// Split of an n x m problem; `abs`: the float64 log form over a resident K.
// Returns false when the shape does not fit the kernel.
template <typename T>
bool fu_plan(int64_t n, int64_t m, bool abs, int grid, const FuDevice& d, FuPlan& f) {
  constexpr int W = Vec<T>::N;
  const int64_t V = (m + W - 1) / W;        // vectors of a row
  if (V > (int64_t)FU_WARPS * 32 * 16 || n > 0x7fffff00) return false;
  f.grid = grid;
  const int64_t rows = (n + grid - 1) / grid;
  auto split = [&](int nk) {
    f.NK = nk;
    f.G = 1;
    while (f.G < FU_WARPS && (int64_t)f.G * 32 * nk < V) f.G *= 2;
    f.kv = nk;
    f.mp = nk * f.G * 32 * W;
    const int NG = FU_WARPS / f.G;
    f.buf_elems = NG > 1 ? std::max(NG * f.mp, FU_WARPS * 32) : 0;
    return (int64_t)f.G * 32 * nk >= V;
  };
  f.NC = 0;
  for (int nk : {1, 2, 3, 4, 6, 8, 12, 16}) {
    if (!split(nk)) continue;
    const size_t tile = sizeof(T) * (size_t)rows * f.mp;
    f.smem = sizeof(T) * ((size_t)f.mp * (abs ? 2 : 1) + f.buf_elems) + tile;
    f.res = rows <= 65536 && f.smem + fu_static_smem<T>(nk) <= d.smem;
    if (f.res) return true;
  }
  if (abs) return false;
  // a row's vectors beyond its end cost as much as the others: 4100 floats
  // (1025 vectors, 9 per thread) took 27.1 us per pass over 3001 rows with
  // NK = 16.  With up to 8 per thread the second half of 16 is left out.
  split(16);
  const int need = (int)((V + f.G * 32 - 1) / (f.G * 32)), nk = need <= 8 ? 16 : std::max(10, (need + 1) / 2 * 2);
  f.NK = nk;
  f.mp = nk * f.G * 32 * W;
  f.buf_elems = FU_WARPS / f.G > 1 ? std::max(FU_WARPS / f.G * f.mp, FU_WARPS * 32) : 0;
  f.kv = need;
  const size_t half = sizeof(T) * (size_t)(FU_WARPS / f.G) * (f.mp / 2);  // 20 to 32 KB over the groups
  for (f.NC = FU_RING; f.NC >= 4; --f.NC) {
    f.smem = sizeof(T) * ((size_t)f.mp + f.buf_elems) + f.NC * half + 16 * ((size_t)(FU_WARPS / f.G * f.NC + 1) / 2);
    if (f.smem + fu_static_smem<T>(nk) <= d.smem) return true;
  }
  return false;
}

constexpr size_t FU_PACK_MAX = (size_t)16 << 30;

// Workspace: published words, pairs, fallback v, padded rows.
struct FuSpace { size_t part, vll, stll, ell, pairs, vfix, mass, pack, total; };
template <typename T>
FuSpace fu_space(int64_t n, int64_t m, int grid, const FuDevice& d) {
  FuSpace w{};
  size_t off = 0;
  auto take = [&](size_t b) { const size_t o = off; off += (b + 255) / 256 * 256; return o; };
  FuPlan f, g;
  if (!fu_plan<T>(n, m, false, grid, d, f)) return w;
  w.part = take(8 * (size_t)Ll<T>::N * grid * m);
  w.vll = take(8 * (size_t)Ll<T>::N * m);
  w.stll = take(8 * (size_t)grid);
  w.ell = take(96 * (size_t)grid);
  w.pairs = take(2 * sizeof(T) * (size_t)grid * m);
  w.vfix = take(sizeof(T) * (size_t)m);
  w.mass = take(8 * (size_t)grid);
  w.pack = off;
  const bool streamed = !f.res || (sizeof(T) == 8 && !fu_plan<T>(n, m, true, grid, d, g));
  if (streamed && m % Vec<T>::N) {
    const size_t b = sizeof(T) * (size_t)n * ((m + Vec<T>::N - 1) / Vec<T>::N * Vec<T>::N);
    if (b > FU_PACK_MAX) return FuSpace{};
    take(b);
  }
  w.total = off;
  return w;
}

template <typename T, int MODE, int NK, bool RES>
int fu_start(FusedArgs<T>& A, const FuPlan& f, cudaStream_t st) {
  const void* k = (const void*)fused_sinkhorn_kernel<T, MODE, NK, RES>;
  if (!allow_smem(k, f.smem)) return OTG_ERR_UNSUPPORTED;
  void* args[] = {&A};
  return cudaLaunchCooperativeKernel(k, dim3(f.grid), dim3(FU_THREADS), args, f.smem, st) == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}

template <typename T, int MODE>
int fu_start_resident(FusedArgs<T>& A, const FuPlan& f, cudaStream_t st) {
  switch (f.NK) {
    case 1: return fu_start<T, MODE, 1, true>(A, f, st);
    case 2: return fu_start<T, MODE, 2, true>(A, f, st);
    case 3: return fu_start<T, MODE, 3, true>(A, f, st);
    case 4: return fu_start<T, MODE, 4, true>(A, f, st);
    case 6: return fu_start<T, MODE, 6, true>(A, f, st);
    case 8: return fu_start<T, MODE, 8, true>(A, f, st);
    case 12: return fu_start<T, MODE, 12, true>(A, f, st);
    default: return fu_start<T, MODE, 16, true>(A, f, st);
  }
}

template <typename T, int MODE>
int fu_start_streamed(FusedArgs<T>& A, const FuPlan& f, cudaStream_t st) {
  switch (f.NK) {
    case 10: return fu_start<T, MODE, 10, false>(A, f, st);
    case 12: return fu_start<T, MODE, 12, false>(A, f, st);
    case 14: return fu_start<T, MODE, 14, false>(A, f, st);
    default: return fu_start<T, MODE, 16, false>(A, f, st);
  }
}

// The launches by mode and type, split over translation units.
template <typename T> int fu_launch_log(FusedArgs<T>& A, const FuPlan& f, bool abs, cudaStream_t st);
template <typename T> int fu_launch_scal(FusedArgs<T>& A, const FuPlan& f, cudaStream_t st);
template <typename T> int fu_launch_unb(FusedArgs<T>& A, const FuPlan& f, cudaStream_t st);

inline int fu_mode(const OtgDenseProblem* p) {
  return p->method == OTG_METHOD_LOG ? FU_LOG : p->method == OTG_METHOD_KNOPP ? FU_SCAL : p->method == OTG_METHOD_UNB ? FU_UNB : -1;
}

template <typename T>
bool fu_choose(const OtgDenseProblem* p, int& mode, const FuDevice& d, FuPlan& f) {
  mode = fu_mode(p);
  if (mode < 0) return false;
  const int grid = fu_grid<T>(p->n, p->m, p->grid, d.sms);
  if (sizeof(T) == 8 && mode == FU_LOG && fu_plan<T>(p->n, p->m, true, grid, d, f)) { mode = FU_ABS; return true; }
  return fu_plan<T>(p->n, p->m, false, grid, d, f);
}

template <typename T>
int fused_run(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st) {
  const FuDevice d = fu_device();
  FuPlan f;
  int mode;
  if (!fu_choose<T>(p, mode, d, f)) return OTG_ERR_UNSUPPORTED;
  constexpr int W = Vec<T>::N;
  FusedArgs<T> A{};
  const bool useK = p->method == OTG_METHOD_KNOPP && p->K;
  A.M = static_cast<const T*>(useK ? p->K : p->M);
  A.n = (int)p->n; A.m = (int)p->m; A.ldm = useK ? p->ldk : p->ldm;
  A.c = (T)(-OTG_LOG2E / p->reg);
  A.mv = (int)((p->m + W - 1) / W * W);
  A.gvec = p->m % W == 0 && A.ldm % W == 0 && (uintptr_t)A.M % 16 == 0;
  const FuSpace w = fu_space<T>(p->n, p->m, f.grid, d);
  char* base = static_cast<char*>(fs.space);
  A.kmat = useK;
  if (!f.res && !A.gvec) {
    if (p->m % W == 0) return OTG_ERR_UNSUPPORTED;  // whole vectors at an odd address or stride: no room set aside
    T* out = reinterpret_cast<T*>(base + w.pack);
    const bool expo = mode != FU_LOG && !useK;
    const T pad = mode != FU_LOG ? T(0) : (A.c > T(0) ? T(-INFINITY) : T(INFINITY));
    const int blocks = (int)std::min<int64_t>(p->n, (int64_t)d.sms * 8);
    fused_pack_kernel<T><<<blocks, 256, 0, st>>>(A.M, p->n, p->m, A.ldm, A.c, expo, pad, out, A.mv);
    if (cudaGetLastError() != cudaSuccess) return OTG_ERR_CUDA;
    A.M = out; A.ldm = A.mv; A.gvec = 1;
    if (mode != FU_LOG) A.kmat = 1;
  }
  A.a = static_cast<const T*>(p->a); A.b = static_cast<const T*>(p->b);
  A.warm_u = static_cast<const T*>(p->warm_u); A.warm_v = static_cast<const T*>(p->warm_v);
  A.max_iter = p->max_iter; A.stop_thr = p->stop_thr; A.period = 10;
  A.u0 = (T*)fs.u0; A.u1 = (T*)fs.u1; A.v0 = (T*)fs.v0; A.v1 = (T*)fs.v1; A.rowc = (T*)fs.rowc; A.fref = (T*)fs.fref;
  A.part = (unsigned long long*)(base + w.part); A.vll = (unsigned long long*)(base + w.vll);
  A.stll = (unsigned long long*)(base + w.stll); A.ell = (unsigned long long*)(base + w.ell);
  A.pairs = (T*)(base + w.pairs); A.vfix = (T*)(base + w.vfix);
  A.mass = (double*)(base + w.mass);
  A.out_u = (T*)p->out_u; A.out_v = (T*)p->out_v;
  A.hist = fs.hist; A.hist_cap = p->hist_cap; A.info = fs.info; A.bar = fs.bar;
  A.timeout_ns = fs.timeout_ns;
  A.G = f.G; A.kv = f.kv; A.mp = f.mp; A.NC = f.NC; A.buf_elems = f.buf_elems;
  if (mode == FU_UNB) {
    A.fi1 = (T)(std::isinf(p->reg_m1) ? 1.0 : p->reg_m1 / (p->reg_m1 + p->reg));
    A.fi2 = (T)(std::isinf(p->reg_m2) ? 1.0 : p->reg_m2 / (p->reg_m2 + p->reg));
    A.alw = p->c_ones ? nullptr : A.a;
    A.bew = p->c_ones ? nullptr : A.b;
    return fu_launch_unb<T>(A, f, st);
  }
  if (mode == FU_SCAL) return fu_launch_scal<T>(A, f, st);
  return fu_launch_log<T>(A, f, mode == FU_ABS, st);
}

template <typename T>
size_t fused_run_bytes(int64_t n, int64_t m, int requested_grid) {
  const FuDevice d = fu_device();
  return fu_space<T>(n, m, fu_grid<T>(n, m, requested_grid, d.sms), d).total;
}

template <typename T>
bool fused_run_holds_gibbs(const OtgDenseProblem* p) {
  FuPlan f;
  int mode;
  return fu_choose<T>(p, mode, fu_device(), f) && (f.res || p->m % Vec<T>::N != 0);
}

}  // namespace otg
