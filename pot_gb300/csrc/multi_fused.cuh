// Batched Sinkhorn with ONE read of the cost blocks per iteration (included
// by multi.cu; the iteration, the stop tests and the outputs are those of
// multi_sinkhorn_kernel).
//
// As in the dense solver (fused_impl.cuh) a row's entries, exponentiated once
// for the row update, also give its share of the next column update, so an
// iteration is
//   pass   rows of all active problems -> u, column sums        | grid barrier
//   merge  column sums -> next v, marginal errors               | grid barrier
//   [checks: problems leave, the active list is rebuilt; Anderson mixing]
// with half the reads and half the exponentials of a column pass followed by
// a row pass (256 blocks of 2048 x 2048 float32: two passes of 0.70 ms each
// before).
//
// Split.  The rows of the active problems, weighted by their width, are cut
// into equal contiguous shares, one per worker: G warps that hold a row
// between them (G = 1 up to 512 16-byte vectors, i.e. 2048 floats, so that
// nothing but the shuffles of one warp stands between a row and its column
// sums).  A lane holds NK vectors of each of RB rows, 256 bytes in all, as in
// the dense kernel: rows of 512 floats go four at a time through one bulk
// copy, one reduction and one division (128 blocks of 512 x 512: 83 us per
// iteration one row at a time).  A worker goes through its share problem by problem: v of the
// problem into shared memory, rows through a ring of bulk copies that runs
// ahead over problem and iteration borders, column sums in registers, and at
// the border of a problem the sums go to the worker's slot of that problem.
// Slots are laid out so that no two overlap: problem k's columns at
// (columns before k) + worker * (widest problem).  Workers are numbered
// across the SMs first, and a batch of few rows uses fewer workers (eight
// rows each), as every worker adds a slot to each column's merge.
#pragma once
#include <type_traits>
#include "fused_ops.cuh"

namespace otg {

constexpr int MF_RING = 4;  // most batches in flight per worker

struct MfRing { int slot; uint32_t phase; bool primed; };

// A worker's share and place in it: problem slot k, rows [row, end) of it.
struct MfSpan { int k, row, end; };

// Cost of a row in a kernel of NK vectors per lane, in vectors.  A batch of
// rows costs its chain of latencies whatever the width, then float32 its
// bytes: per row 0.42 ns at 64 floats, 0.46 at 512, 0.68 at 1024 with NK = 8
// (0.15 to 0.22 with NK = 2, 0.81 to 1.29 with 16).  float64 costs the
// exponentials of the half or all of the NK vectors that are evaluated: 6.8
// and 11.6 ns with NK = 4.  (Weights in proportion to the width left the
// worker with the narrowest rows 2.2 times the mean on 256 ragged blocks.)
template <typename T>
__device__ __forceinline__ int mf_weight(const MultiArgs<T>& A, int ldm) {
  const int nv = ldm / Vec<T>::N;
  if (sizeof(T) == 8) return 2 * nv > A.fNK * A.fG * 32 ? 40 * A.fNK : 24 * A.fNK;
  return nv + 45 * A.fNK * A.fG;
}

// Share [beg, end) of worker w in weight units.
__device__ __forceinline__ void mf_range(int64_t total, int w, int na, int64_t& beg, int64_t& end) {
  beg = total * w / na;
  end = total * (w + 1) / na;
}
// The worker whose share holds weight position `pos`.
__device__ __forceinline__ int mf_worker(int64_t total, int na, int64_t pos) {
  int w = (int)min((int64_t)(na - 1), pos * na / total);
  while (w > 0 && total * w / na > pos) --w;
  while (w + 1 < na && total * (w + 1) / na <= pos) ++w;
  return w;
}

// Rows of slot k in the share [beg, end): whole batches, those that start in
// it (shares cut at any row had up to two partial batches more).
template <typename T>
__device__ __forceinline__ MfSpan mf_span(const MultiArgs<T>& A, int k, int64_t beg, int64_t end) {
  const int p = __ldcg(A.active + k);
  const int64_t base = __ldcg(A.urow_pre + k);
  const int wt = mf_weight(A, A.ldm[p]), n = A.rows[p];
  const int64_t bw = (int64_t)wt * (16 / A.fNK);
  MfSpan s;
  s.k = k;
  s.row = beg <= base ? 0 : (int)min((int64_t)n, (beg - base + bw - 1) / bw * (16 / A.fNK));
  s.end = end <= base ? 0 : (int)min((int64_t)n, (end - base + bw - 1) / bw * (16 / A.fNK));
  return s;
}
// First span of a share, and the one behind a span (k = nact: none).
template <typename T>
__device__ __forceinline__ MfSpan mf_next(const MultiArgs<T>& A, int k, int nact, int64_t beg, int64_t end) {
  for (; k < nact && __ldcg(A.urow_pre + k) < end; ++k) {
    const MfSpan s = mf_span(A, k, beg, end);
    if (s.row < s.end) return s;
  }
  return MfSpan{nact, 0, 0};
}

// What a worker needs of a problem in its share.  The first MF_KEPT of them
// are kept in shared memory until the shares change: looked up anew they cost
// a chain of some ten loads from L2 in every pass (6 us).
constexpr int MF_KEPT = 6;
template <typename T>
struct MfPart {
  int64_t ro, co;   // offsets of a / u and of b / v
  int64_t out;      // worker's slot of the column sums
  T c;
  int k, row, end, p, m, ldm;
};
template <typename T>
__device__ __forceinline__ MfPart<T> mf_part(const MultiArgs<T>& A, const MfSpan& s, int w) {
  MfPart<T> q;
  q.k = s.k; q.row = s.row; q.end = s.end;
  q.p = __ldcg(A.active + s.k);
  q.m = A.cols[q.p]; q.ldm = A.ldm[q.p];
  q.ro = A.r_off[q.p]; q.co = A.c_off[q.p];
  q.out = __ldcg(A.ucol_pre + s.k) + (int64_t)w * A.fmm;
  q.c = (T)(-OTG_LOG2E / A.reg[q.p]);
  return q;
}

// Ring cursor (one lane per worker): the next batch to copy.
template <typename T>
struct MfCursor {
  MfSpan s;
  const T* src;
  int ldm;
};
template <typename T>
__device__ __forceinline__ void mf_cursor(const MultiArgs<T>& A, MfCursor<T>& c) {
  const int p = __ldcg(A.active + c.s.k);
  c.ldm = A.ldm[p];  // padded columns hold +inf: copied as they are
  c.src = A.M + A.m_off[p] + (int64_t)c.s.row * c.ldm;
}
// The cursor's batch (up to RB adjacent rows) in one copy; on to the next one
// (behind the last: the first again, for the next iteration).
template <typename T, int RB>
__device__ __forceinline__ void mf_issue(const MultiArgs<T>& A, MfCursor<T>& c, T* dst, uint64_t* full, int k0, int nact, int64_t beg,
                                         int64_t end) {
  const int rows = min(RB, c.s.end - c.s.row);
  const uint32_t bytes = (uint32_t)(rows * c.ldm) * (uint32_t)sizeof(T);
  mbar_arrive_expect_tx(full, bytes);
  bulk_g2s(dst, c.src, bytes, full);
  c.src += (int64_t)RB * c.ldm;
  c.s.row += RB;
  if (c.s.row >= c.s.end) {
    c.s = mf_next(A, c.s.k + 1, nact, beg, end);
    if (c.s.k == nact) c.s = mf_next(A, k0, nact, beg, end);
    mf_cursor(A, c);
  }
}

template <typename T>
struct MfSmem { T* vs; T* data; uint64_t* full; MfPart<T>* kept; };

// A worker's share (the same in every lane until the active list changes).
struct MfShare { int64_t beg, end; int k0, kept; };

__device__ __forceinline__ void mf_sync(const FuRow& R, int G) {
  if (G == 1) __syncwarp(); else named_bar(1 + R.g, R.gt);
}

// v of one problem into the worker's shared copy, `pad` beyond the row.
template <typename T>
__device__ __forceinline__ void mf_load_v(const FuRow& R, int G, T* vs, const T* v, int m, int mp, T pad) {
  using V = typename Vec<T>::type;
  constexpr int W = Vec<T>::N, U = 16;
  mf_sync(R, G);  // the previous problem's v has been read
  int j = R.tg;
  if (((uintptr_t)v & 15) == 0) {
    const int nv = m / W;
    for (; j < nv; j += U * R.gt) {
      V x[U];
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (j + q * R.gt < nv) x[q] = __ldcg(reinterpret_cast<const V*>(v) + j + q * R.gt);
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (j + q * R.gt < nv) reinterpret_cast<V*>(vs)[j + q * R.gt] = x[q];
    }
    j = nv * W + R.tg;
  } else {
    for (; j + (U - 1) * R.gt < m; j += U * R.gt) {
      T x[U];
#pragma unroll
      for (int q = 0; q < U; ++q) x[q] = __ldcg(v + j + q * R.gt);
#pragma unroll
      for (int q = 0; q < U; ++q) vs[j + q * R.gt] = x[q];
    }
  }
  for (; j < mp; j += R.gt) vs[j] = j < m ? __ldcg(v + j) : pad;
  mf_sync(R, G);
}

// The share of worker w, its first problems kept.
template <typename T>
__device__ __noinline__ MfShare mf_share(const MultiArgs<T>& A, const FuRow& R, MfPart<T>* kept, int w, int na, int nact) {
  MfShare S;
  mf_range(__ldcg(A.urow_pre + nact), w, na, S.beg, S.end);
  S.k0 = mt_find(A.urow_pre, nact, S.beg);
  S.kept = 0;
  for (MfSpan s = mf_next(A, S.k0, nact, S.beg, S.end); s.k < nact && S.kept < MF_KEPT; s = mf_next(A, s.k + 1, nact, S.beg, S.end)) {
    const MfPart<T> q = mf_part(A, s, w);
    if (R.tg == 0) kept[S.kept] = q;
    ++S.kept;
  }
  return S;
}

// One pass over a worker's share.
template <typename T, bool LOGF, int NK>
__device__ __forceinline__ bool mf_pass(const MultiArgs<T>& A, const FuRow& R, const MfSmem<T>& sm, T (*red)[FU_WARPS][1], MfRing& ring,
                                        MfCursor<T>& cur, const MfShare& S, int w, int nact, const T* v) {
  using V = FuV<T>;
  constexpr int W = Vec<T>::N, RB = 16 / NK, LPR = 32 / RB;
  const int64_t beg = S.beg, end = S.end;
  const int G = RB > 1 ? 1 : A.fG, nc = A.fNC, mp = A.fmp;  // a row of several warps goes alone
  const int chunk = RB * mp;
  const uint32_t hop = (uint32_t)R.gt * 16u;
  const uint32_t va = smem_addr(sm.vs) + (uint32_t)R.tg * 16u, xa = smem_addr(sm.data) + (uint32_t)R.tg * 16u;
  const int k0 = S.k0;
  if (!ring.primed) {
    ring.primed = true;
    if (R.tg == 0) {
      cur.s = mf_next(A, k0, nact, beg, end);
      mf_cursor(A, cur);
      for (int q = 0; q < nc; ++q) {
        const int sl = ring.slot + q < nc ? ring.slot + q : ring.slot + q - nc;
        mf_issue<T, RB>(A, cur, sm.data + sl * chunk, sm.full + sl, k0, nact, beg, end);
      }
    }
  }
  bool ok = true;
  int par = 0;
  const int myrow = R.lane / LPR;  // row of the batch that this lane finishes
  for (int at_part = 0, k_last = -1;; ++at_part) {
    MfPart<T> s;
    if (at_part < S.kept) {
      s = sm.kept[at_part];
    } else {
      if (S.kept < MF_KEPT) break;
      const MfSpan sp = mf_next(A, k_last + 1, nact, beg, end);
      if (sp.k == nact) break;
      s = mf_part(A, sp, w);
    }
    k_last = s.k;
    const int ldm = s.ldm, nv = ldm / W;
    const int64_t ro = s.ro;
    const typename V::S c = V::all(s.c);
    mf_load_v(R, G, sm.vs, v + s.co, s.m, mp, LOGF ? T(-INFINITY) : T(0));
    const bool wide = nv > (NK / 2) * R.gt;  // more than NK / 2 vectors per lane
    const uint32_t pitch = (uint32_t)ldm * (uint32_t)sizeof(T);
    V acc[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) acc[k] = V::zero();
    T q0 = 0, q1 = 0, q2 = 0;  // u, log2 a, a of row `lane` of the 32 in hand
    for (int row = s.row; row < s.end; row += RB) {
      const int at = (row - s.row) & 31, nr = min(RB, s.end - row);
      if (at == 0) {
        const int64_t i = ro + row + R.lane;
        if (row + R.lane < s.end) {
          q0 = __ldcg(A.u + i);
          q2 = A.a[i];
          if (LOGF) q1 = lg2(q2);
        }
      }
      V e[RB][NK];
      T sum[RB];
      if (!mbar_wait(sm.full + ring.slot, ring.phase, A.ctl + 1, A.timeout_ns)) ok = false;
      const uint32_t xb = xa + (uint32_t)(ring.slot * chunk) * (uint32_t)sizeof(T);
      // Loads and exponentials of a batch in one block of code (no branch per
      // vector or row).  Rows beyond the batch read its last one again and
      // nothing comes of them; vectors beyond the row (`tail`: there are
      // some) count as zeros against a v that adds nothing.
      auto eval = [&](auto kv, auto tail) {
        constexpr int KV = decltype(kv)::value;
        constexpr bool TAIL = decltype(tail)::value;
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          const uint32_t xq = xb + (uint32_t)min(q, nr - 1) * pitch;
          const typename V::S h = V::all(LOGF ? __shfl_sync(0xffffffffu, q2 == T(0) ? T(-INFINITY) : q0 - q1, at + q) : T(0));
          V t4 = V::zero();
#pragma unroll
          for (int k = 0; k < KV; ++k) {
            const V vv = V::lds(va + k * hop);
            // (wide rows: the first half of the vectors is full)
            const V x = TAIL && (KV < NK || k >= NK / 2) ? V::lds_if(xq + k * hop, k * R.gt + R.tg < nv) : V::lds(xq + k * hop);
            if (LOGF) { e[q][k] = V::expo(x, c, vv, h); t4.add_v(e[q][k]); }
            else { e[q][k] = V::gibbs(x, c); t4.fma_v(e[q][k], vv); }
          }
#pragma unroll
          for (int k = KV; k < NK; ++k) e[q][k] = V::zero();
          sum[q] = t4.sum();
        }
      };
      using Kall = std::integral_constant<int, NK>;
      using Khalf = std::integral_constant<int, NK / 2>;
      if (wide) { if (nv == NK * R.gt) eval(Kall{}, std::false_type{}); else eval(Kall{}, std::true_type{}); }
      else { if (nv == NK / 2 * R.gt) eval(Khalf{}, std::false_type{}); else eval(Khalf{}, std::true_type{}); }
      T t;
      if constexpr (RB == 1) t = fu_group<T, 1, false>(sum, R, G, red, par);
      else t = fu_scatter<T, RB, false>(sum, R.lane);
      const T uo = __shfl_sync(0xffffffffu, q0, at + myrow), ai = __shfl_sync(0xffffffffu, q2, at + myrow);
      T un, r;
      if constexpr (LOGF) {
        // a row of no weight adds nothing to any column
        const bool none = ai == T(0);
        if (none) t = T(1);
        un = uo - lg2(t);
        r = ai / t;
        if (A.relax) { un = fma(A.omega, un - uo, uo); r = ai * ex2(un - uo); }
        if (none) { un = T(-INFINITY); r = T(0); }
        if (!__all_sync(0xffffffffu, myrow >= nr || fu_near_one(t))) {
          // running maxima, on the same entries (the slot is not refilled yet)
          T mx[RB];
#pragma unroll
          for (int q = 0; q < RB; ++q) {
            mx[q] = -INFINITY;
            const uint32_t xq = xb + (uint32_t)min(q, nr - 1) * pitch;
#pragma unroll
            for (int k = 0; k < NK; ++k)
              if (k < NK / 2 || wide) { e[q][k] = V::arg(V::lds_if(xq + k * hop, k * R.gt + R.tg < nv), c, V::lds(va + k * hop)); mx[q] = e[q][k].max_with(mx[q]); }
          }
          T mg;
          if constexpr (RB == 1) mg = fu_group<T, 1, true>(mx, R, G, red, par);
          else mg = fu_scatter<T, RB, true>(mx, R.lane);
#pragma unroll
          for (int q = 0; q < RB; ++q) {
            const T mq = __shfl_sync(0xffffffffu, mg, q * LPR);
            V t5 = V::zero();
#pragma unroll
            for (int k = 0; k < NK; ++k)
              if (k < NK / 2 || wide) { e[q][k] = V::ex_minus(e[q][k], mq); t5.add_v(e[q][k]); }
            sum[q] = t5.sum();
          }
          if constexpr (RB == 1) t = fu_group<T, 1, false>(sum, R, G, red, par);
          else t = fu_scatter<T, RB, false>(sum, R.lane);
          const T la = __shfl_sync(0xffffffffu, q1, at + myrow);
          un = la - lse_value(mg, t);
          r = ai / t;
          if (A.relax) { un = fma(A.omega, un - uo, uo); r = ex2(un + mg); }
          if (none) { un = T(-INFINITY); r = T(0); }
        }
      } else {
        un = ai / t;
        r = un;
      }
      __syncwarp();  // (groups of several warps: the reductions' barriers) the slot has been read
      if (R.tg == 0) mf_issue<T, RB>(A, cur, sm.data + ring.slot * chunk, sm.full + ring.slot, k0, nact, beg, end);
      if (++ring.slot == nc) { ring.slot = 0; ring.phase ^= 1; }
      {
        const int mine = R.lane - at;
        const T x = __shfl_sync(0xffffffffu, un, (mine >= 0 && mine < RB ? mine : 0) * LPR);
        if (mine >= 0 && mine < nr) q0 = x;
      }
      if ((at + RB == 32 || row + RB >= s.end) && R.tg < at + nr && R.tg < 32) A.u[ro + row - at + R.lane] = q0;
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        const typename V::S rs = V::all(__shfl_sync(0xffffffffu, r, q * LPR));
        if (q < nr) {
#pragma unroll
          for (int k = 0; k < NK; ++k) acc[k].fma_s(e[q][k], rs);
        }
      }
    }
    // the worker's column sums of this problem
    T* dst = A.fpart + s.out;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const int j = k * R.gt + R.tg;
      if (j < nv) {
        T x[W];
        acc[k].get(x);
        fu_put(dst + j * W, x);
      }
    }
  }
  return ok;
}

// Column log-sum-exp pairs (LOGF) or column sums of u alone over a worker's
// share: the first v, and (MARKED) the columns whose `marks` is NaN of problems
// flagged in A.fbad.
template <typename T, bool LOGF, bool MARKED>
__device__ __noinline__ void mf_colpass(const MultiArgs<T>& A_, const FuRow& R_, int w, int na, int nact, const T* marks) {
  constexpr int W = Vec<T>::N, KB = MARKED ? 1 : 4, RW = 16 / KB;
  const MultiArgs<T> A = A_;
  const FuRow R = R_;
  const int64_t total = __ldcg(A.urow_pre + nact);
  int64_t beg, end;
  mf_range(total, w, na, beg, end);
  for (MfSpan sp = mf_next(A, mt_find(A.urow_pre, nact, beg), nact, beg, end); sp.k < nact; sp = mf_next(A, sp.k + 1, nact, beg, end)) {
    const int p = __ldcg(A.active + sp.k);
    if (MARKED && __ldcg(A.fbad + p) == 0) continue;
    const int ldm = A.ldm[p], nv = ldm / W, m = A.cols[p];
    const int64_t co = A.c_off[p];
    const T c = (T)(-OTG_LOG2E / A.reg[p]);
    const T* Mp = A.M + A.m_off[p];
    const T* up = A.u + A.r_off[p];
    const int64_t at = __ldcg(A.ucol_pre + sp.k) + (int64_t)w * A.fmm;
    for (int k0 = 0; k0 * R.gt < nv; k0 += KB) {
      T mx[KB][W], s[KB][W];
#pragma unroll
      for (int k = 0; k < KB; ++k)
#pragma unroll
        for (int x = 0; x < W; ++x) { mx[k][x] = -INFINITY; s[k][x] = 0; }
      bool on = true;
      if (MARKED) {
        const int j = k0 * R.gt + R.tg;
        on = false;
#pragma unroll
        for (int x = 0; x < W; ++x) on |= j * W + x < m && isnan(__ldcg(marks + co + j * W + x));
      }
      for (int row = on ? sp.row : sp.end; row < sp.end; row += RW) {
        T ui[RW];
#pragma unroll
        for (int q = 0; q < RW; ++q) ui[q] = row + q < sp.end ? __ldcg(up + row + q) : (LOGF ? T(-INFINITY) : T(0));
        // sixteen loads in flight at once (vectors beyond the row read its
        // first one and are not stored)
        T x[KB][RW][W];
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const int j = (k0 + k) * R.gt + R.tg < nv ? (k0 + k) * R.gt + R.tg : 0;
#pragma unroll
          for (int q = 0; q < RW; ++q)
            unpack(ld_stream(reinterpret_cast<const typename Vec<T>::type*>(Mp + (int64_t)min(row + q, sp.end - 1) * ldm) + j), x[k][q]);
        }
#pragma unroll
        for (int k = 0; k < KB; ++k) {
#pragma unroll
          for (int y = 0; y < W; ++y) {
            if (LOGF) {
              // rows beyond the share have u = -inf
              T t[RW], top = mx[k][y];
#pragma unroll
              for (int q = 0; q < RW; ++q) { t[q] = row + q < sp.end ? fma(x[k][q][y], c, ui[q]) : T(-INFINITY); top = fmax(top, t[q]); }
              // (an empty column so far: the sums stay zero)
              const T ref = top == -INFINITY ? T(0) : top;
              T sum = s[k][y] * ex2(mx[k][y] - ref);
#pragma unroll
              for (int q = 0; q < RW; ++q) sum += ex2(t[q] - ref);
              s[k][y] = sum;
              mx[k][y] = top;
            } else {
#pragma unroll
              for (int q = 0; q < RW; ++q) s[k][y] = fma(ex2(x[k][q][y] * c), ui[q], s[k][y]);
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        const int j = (k0 + k) * R.gt + R.tg;
        if (j < nv && on) {
#pragma unroll
          for (int y = 0; y < W; ++y) {
            if (LOGF) {
              A.fpairs[2 * (at + j * W + y)] = mx[k][y];
              A.fpairs[2 * (at + j * W + y) + 1] = s[k][y];
            } else {
              A.fpart[at + j * W + y] = s[k][y];
            }
          }
        }
      }
    }
  }
}

// Merge over 32-column blocks of the active problems: the slots of a column
// are added in worker order, a block per warp, or (`split`) the 8 warps of a
// CTA share a block's slots (their sums in warp order).  The place of the
// first block (looked up once until the shares change) is in `P`.
// fin(p, cj, b, v, mx, s, lim) finishes column cj (packed like b) of problem
// p.  `marks`: only the columns whose mark is NaN, of problems in A.fbad.
// Column sums below 2^lim may have lost bits to underflow (as in fused_impl.cuh,
// a part of the problem's mass).
struct MfPlace { int64_t lo, hi, base, co, b0, b1; int k, p, m, w0, w1, split, lim; };

// A block costs a warp about 1.0 us for its place, v and b and 0.6 us per eight
// slots, all of it latency; split, the CTA 1.3 us and an eighth of the slots.
// The split pays for few blocks with many slots (one problem of 1024 columns:
// 130 slots) and loses as soon as a CTA has many blocks (256 problems of 512
// columns, 7 slots: 27 blocks per CTA, 36 of 78 us per iteration).
__device__ __forceinline__ bool mf_split(int64_t blocks, int na, int nact, int ctas) {
  const int64_t r = (na / nact + 1 + 7) / 8;
  return ((blocks + ctas - 1) / ctas) * (13 + 6 * r / FU_WARPS) < ((blocks + ctas * FU_WARPS - 1) / (ctas * FU_WARPS)) * (10 + 6 * r);
}
template <typename T>
__device__ __forceinline__ void mf_place(const MultiArgs<T>& A, MfPlace& P, int64_t blk, int na, int nact) {
  MtSlot sl{P.k, P.lo, P.hi};
  if (!sl.seek(A.colpre, nact, blk)) return;
  P.k = sl.k; P.lo = sl.lo; P.hi = sl.hi;
  P.p = __ldcg(A.active + P.k);
  P.m = A.cols[P.p];
  P.co = A.c_off[P.p];
  P.lim = __ldcg(A.flim + P.p);
  const int64_t pos = __ldcg(A.urow_pre + P.k), total = __ldcg(A.urow_pre + nact);
  P.w0 = mf_worker(total, na, pos);
  const int rb = 16 / A.fNK;  // the last batch's place
  P.w1 = mf_worker(total, na, pos + (int64_t)((A.rows[P.p] - 1) / rb * rb) * mf_weight(A, A.ldm[P.p]));
  P.base = __ldcg(A.ucol_pre + P.k);
}
template <typename T>
__device__ __noinline__ MfPlace mf_first_place(const MultiArgs<T>& A, int na, int nact) {
  const int64_t blocks = __ldcg(A.colpre + nact);
  MfPlace P{};
  P.split = mf_split(blocks, na, nact, gridDim.x);
  if (P.split) mt_share(blocks, blockIdx.x, gridDim.x, P.b0, P.b1);
  else mt_share(blocks, (long)blockIdx.x * FU_WARPS + (threadIdx.x >> 5), (long)gridDim.x * FU_WARPS, P.b0, P.b1);
  P.k = -1;
  if (P.b0 < P.b1) mf_place(A, P, P.b0, na, nact);
  return P;
}
template <typename T, bool PAIRS, typename Fin>
__device__ __forceinline__ void mf_merge(const MultiArgs<T>& A, const MfPlace& first, int na, int nact, T (*scr)[2][32], const T* marks,
                                         const T* vcur, Fin&& fin) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  MfPlace P = first;
  const bool split = P.split;
  for (int64_t blk = P.b0; blk < P.b1; ++blk) {
    mf_place(A, P, blk, na, nact);
    if (marks && __ldcg(A.fbad + P.p) == 0) continue;
    const int j = (int)(blk - P.lo) * 32 + lane;
    T mx = -INFINITY, s = 0, bj = 0, vo = 0;
    const int step = split ? FU_WARPS : 1;
    bool on = j < P.m;
    if (marks && on) on = isnan(__ldcg(marks + P.co + j));
    if (on) {
      bj = A.b[P.co + j];
      vo = __ldcg(vcur + P.co + j);
      int w = P.w0 + (split ? warp : 0);
      if (PAIRS) {
        if (w <= P.w1)
          lse_merge_strided(mx, s, A.fpairs + 2 * (P.base + (int64_t)w * A.fmm + j), 2 * (int64_t)step * A.fmm, (P.w1 - w) / step + 1);
      } else {
        const T* q = A.fpart + P.base + j;
        for (; w <= P.w1; w += 8 * step) {
          T x[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = w + k * step <= P.w1 ? __ldcg(q + (int64_t)(w + k * step) * A.fmm) : T(0);
#pragma unroll
          for (int k = 0; k < 8; ++k) s += x[k];
        }
      }
    }
    if (split) {
      scr[warp][0][lane] = s;
      scr[warp][1][lane] = mx;
      __syncthreads();
      if (warp == 0) {
        for (int q = 1; q < FU_WARPS; ++q) {
          if (PAIRS) lse_merge(mx, s, scr[q][1][lane], scr[q][0][lane]);
          else s += scr[q][0][lane];
        }
      }
      __syncthreads();
    }
    if (on && (!split || warp == 0)) fin(P.p, P.co + j, bj, vo, mx, s, P.lim);
  }
}

// ---------------------------------------------------------------------------
// Anderson mixing of the next v (anderson.cuh), in three steps between grid
// barriers: dots of the new residual with the history by blocks of 32 columns
// over all warps, the weights by one warp per problem, the mixing by blocks.
// A CTA per problem did the same in 145 us for 256 problems of 2048 columns:
// two problems in a row on most SMs, each a chain of loads and of FP64.  Now
// 100 us: dots 28, weights 20, mixing 23, the barriers and waits the rest.
// ---------------------------------------------------------------------------
constexpr int MF_ANDW = OTG_ANDERSON_MAX_DEPTH + 2;  // weights, whether to mix, slots in use
constexpr int MF_ANDB = 4;                           // blocks of a warp in flight
template <typename T>
__device__ __noinline__ void mf_and_dots(const MultiArgs<T>& A, int nact, const T* vcur, const T* vnxt) {
  constexpr int MD = OTG_ANDERSON_MAX_DEPTH;
  const int lane = threadIdx.x & 31, D = A.and_depth;
  int64_t b0, b1;
  mt_share(__ldcg(A.colpre + nact), (long)blockIdx.x * FU_WARPS + (threadIdx.x >> 5), (long)gridDim.x * FU_WARPS, b0, b1);
  MtSlot sl;
  int64_t co = 0;
  int m = 0, s = 0, nh = 0;
  for (int64_t blk = b0; blk < b1;) {
    if (sl.seek(A.colpre, nact, blk)) {
      const int p = __ldcg(A.active + sl.k), cnt = __ldcg(A.and_cnt + p);
      m = A.cols[p]; co = A.c_off[p];
      s = cnt % D; nh = min(cnt + 1, D);
    }
    const int nb = (int)min((int64_t)MF_ANDB, min(b1, sl.hi) - blk), j0 = (int)(blk - sl.lo) * 32 + lane;
    T f[MF_ANDB], r[MF_ANDB], h[MF_ANDB][MD];
#pragma unroll
    for (int i = 0; i < MF_ANDB; ++i) {
      const int j = j0 + 32 * i;
      const bool on = i < nb && j < m;
      f[i] = on ? __ldcg(vnxt + co + j) : T(0);
      r[i] = on ? __ldcg(vcur + co + j) : T(0);
#pragma unroll
      for (int q = 0; q < MD; ++q) h[i][q] = on && q < nh && q != s ? __ldcg(A.and_R + q * A.total_cols + co + j) : T(0);
    }
    double acc[MD];
#pragma unroll
    for (int q = 0; q < MD; ++q) acc[q] = 0.0;
#pragma unroll
    for (int i = 0; i < MF_ANDB; ++i) {
      const int j = j0 + 32 * i;
      if (i < nb) {
        r[i] = f[i] - r[i];
        if (j < m) {
          A.and_F[s * A.total_cols + co + j] = f[i];
          A.and_R[s * A.total_cols + co + j] = r[i];
        }
        const double rd = widen(r[i]);
#pragma unroll
        for (int q = 0; q < MD; ++q)
          if (q < nh) acc[q] += rd * (q == s ? rd : widen(h[i][q]));
      }
    }
    int o = 16;
#pragma unroll
    for (int g = MD / 2; g >= 1; g /= 2) {
      const bool up = lane & o;
#pragma unroll
      for (int q = 0; q < g; ++q) {
        const double keep = up ? acc[q + g] : acc[q], give = up ? acc[q] : acc[q + g];
        acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      o >>= 1;
    }
    double d = acc[0];
#pragma unroll
    for (int q = 16 / MD; q > 0; q >>= 1) d += __shfl_xor_sync(0xffffffffu, d, q);
    if (lane % (32 / MD) == 0) {
      const int q = lane / (32 / MD);
      A.and_part[blk * MD + q] = d;
      for (int i = 1; i < nb; ++i) A.and_part[(blk + i) * MD + q] = 0.0;
    }
    blk += nb;
  }
}

template <typename T>
__device__ __noinline__ void mf_and_solve(const MultiArgs<T>& A, int nact) {
  constexpr int MD = OTG_ANDERSON_MAX_DEPTH;
  const int lane = threadIdx.x & 31, D = A.and_depth;
  for (int k = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; k < nact; k += gridDim.x * FU_WARPS) {
    const int p = __ldcg(A.active + k), cnt = __ldcg(A.and_cnt + p);
    const int s = cnt % D, nh = min(cnt + 1, D);
    const int64_t lo = __ldcg(A.colpre + k), hi = __ldcg(A.colpre + k + 1);
    double d = 0.0;
    for (int64_t b = lo + lane / MD; b < hi; b += 8 * (32 / MD)) {
      double x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = b + i * (32 / MD) < hi ? __ldcg(A.and_part + (b + i * (32 / MD)) * MD + lane % MD) : 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) d += x[i];
    }
#pragma unroll
    for (int o = MD; o < 32; o *= 2) d += __shfl_xor_sync(0xffffffffu, d, o);
    double w;
    const bool ok = anderson_solve(D, nh, s, d, A.and_G + (int64_t)p * D * D, lane, w);
    double* out = A.and_w + (int64_t)p * MF_ANDW;
    if (lane < MD) out[lane] = w;
    if (lane == 0) {
      out[MD] = ok ? 1.0 : 0.0;
      out[MD + 1] = (double)nh;
      // after a failure the history restarts with the next iterate
      A.and_cnt[p] = ok || nh == 1 ? cnt + 1 : 0;
    }
  }
}

template <typename T>
__device__ __noinline__ void mf_and_mix(const MultiArgs<T>& A, int nact, T* vnxt) {
  constexpr int MD = OTG_ANDERSON_MAX_DEPTH;
  const int lane = threadIdx.x & 31;
  int64_t b0, b1;
  mt_share(__ldcg(A.colpre + nact), (long)blockIdx.x * FU_WARPS + (threadIdx.x >> 5), (long)gridDim.x * FU_WARPS, b0, b1);
  MtSlot sl;
  int64_t co = 0;
  int m = 0, nh = 0;
  double w[MD];
  for (int64_t blk = b0; blk < b1;) {
    if (sl.seek(A.colpre, nact, blk)) {
      const int p = __ldcg(A.active + sl.k);
      m = A.cols[p]; co = A.c_off[p];
      const double* at = A.and_w + (int64_t)p * MF_ANDW;
#pragma unroll
      for (int q = 0; q < MD; ++q) w[q] = __ldcg(at + q);
      nh = __ldcg(at + MD) != 0.0 ? (int)__ldcg(at + MD + 1) : 0;
    }
    const int nb = (int)min((int64_t)MF_ANDB, min(b1, sl.hi) - blk), j0 = (int)(blk - sl.lo) * 32 + lane;
    if (nh > 0) {  // (a plain step keeps F(v))
      T h[MF_ANDB][MD];
#pragma unroll
      for (int i = 0; i < MF_ANDB; ++i)
#pragma unroll
        for (int q = 0; q < MD; ++q)
          h[i][q] = q < nh && i < nb && j0 + 32 * i < m ? __ldcg(A.and_F + q * A.total_cols + co + j0 + 32 * i) : T(0);
#pragma unroll
      for (int i = 0; i < MF_ANDB; ++i) {
        if (i < nb && j0 + 32 * i < m) {
          double v = 0.0;
#pragma unroll
          for (int q = 0; q < MD; ++q)
            if (q < nh) v += w[q] * widen(h[i][q]);
          vnxt[co + j0 + 32 * i] = (T)v;
        }
      }
    }
    blk += nb;
  }
}

// Active list and its prefix sums (one CTA): weights of the rows, padded
// columns, 32-column blocks; the number of workers.
template <typename T>
__device__ __noinline__ void mf_rebuild(const MultiArgs<T>& A, int nact, const int32_t* leaving, int* s_scan, int nworkers) {
  __shared__ int s_base;
  __shared__ int64_t s_wt[4][MT_THREADS / 32], s_run[4];
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  for (int c0 = 0; c0 < nact; c0 += blockDim.x) {
    const int k = c0 + threadIdx.x;
    int p = -1, keep = 0;
    if (k < nact) { p = __ldcg(A.active + k); keep = leaving[p] ? 0 : 1; }
    s_scan[threadIdx.x] = keep;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {
      const int add = threadIdx.x >= o ? s_scan[threadIdx.x - o] : 0;
      __syncthreads();
      s_scan[threadIdx.x] += add;
      __syncthreads();
    }
    const int pos = s_base + s_scan[threadIdx.x] - keep;
    if (keep) A.active[pos] = p;  // compaction never overtakes the reads of this chunk
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_base += s_scan[threadIdx.x];
    __syncthreads();
  }
  if (threadIdx.x < 4) s_run[threadIdx.x] = 0;
  __syncthreads();
  const int na = s_base, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c0 = 0; c0 < na; c0 += blockDim.x) {
    const int k = c0 + threadIdx.x;
    int64_t own[4] = {0, 0, 0, 0};
    if (k < na) {
      const int p = A.active[k], ldm = A.ldm[p];
      own[0] = (int64_t)A.rows[p] * mf_weight(A, ldm);
      own[1] = ldm;
      own[2] = (A.cols[p] + 31) / 32;
      own[3] = A.rows[p];
    }
    int64_t inc[4] = {own[0], own[1], own[2], own[3]};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int64_t up = __shfl_up_sync(0xffffffffu, inc[q], o);
        if (lane >= o) inc[q] += up;
      }
    }
    if (lane == 31)
      for (int q = 0; q < 4; ++q) s_wt[q][wid] = inc[q];
    __syncthreads();
    int64_t before[4] = {s_run[0], s_run[1], s_run[2], s_run[3]};
    for (int w = 0; w < wid; ++w)
      for (int q = 0; q < 4; ++q) before[q] += s_wt[q][w];
    if (k < na) {
      A.urow_pre[k] = before[0] + inc[0] - own[0];
      A.ucol_pre[k] = before[1] + inc[1] - own[1];
      A.colpre[k] = before[2] + inc[2] - own[2];
    }
    __syncthreads();
    if (threadIdx.x < 4)
      for (int w = 0; w < MT_THREADS / 32; ++w) s_run[threadIdx.x] += s_wt[threadIdx.x][w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    A.urow_pre[na] = s_run[0]; A.ucol_pre[na] = s_run[1]; A.colpre[na] = s_run[2];
    int tail = A.tail_max > 0 && na > 0 && na <= A.tail_max;
    for (int k = 0; tail && k < na; ++k) {
      const int p = A.active[k];
      const int64_t rcap = (A.rows[p] + A.tail_cl - 1) / A.tail_cl;
      // rows beyond the shared tile are streamed: up to twice the tile per CTA
      if (A.cols[p] > TL_MAXM || rcap > TL_MAXR || rcap * A.ldm[p] * (int64_t)sizeof(T) > 2 * A.tail_tile) tail = 0;
    }
    // eight rows per worker at least, and a share never lighter than a batch
    // (each worker between a problem's first and last one then has a batch of it)
    int64_t nw = s_run[3] / 8;
    nw = min(nw, s_run[0] / ((int64_t)mf_weight(A, A.fmm) * (16 / A.fNK)));
    nw = max((int64_t)1, min(nw, (int64_t)nworkers));
    A.ctl[7] = (int)nw;
    A.ctl[2] = tail;
    A.ctl[0] = na;
    __threadfence();
  }
  __syncthreads();
}

template <typename T, bool LOGF, int NK>
__global__ void __launch_bounds__(MT_THREADS, 1) multi_fused_kernel(const __grid_constant__ MultiArgs<T> A, int32_t* leaving) {
  extern __shared__ __align__(16) unsigned char mf_smem[];
  __shared__ int s_scan[MT_THREADS];
  __shared__ T red[2][FU_WARPS][1];
  __shared__ T scr[FU_WARPS][2][32];
  __shared__ MfPart<T> s_kept[FU_WARPS][MF_KEPT];
  __shared__ MfShare s_share[FU_WARPS];  // (in shared memory, as registers are what the pass has least of)
  __shared__ MfPlace s_place[FU_WARPS];
  const int G = A.fG;
  FuRow R{};
  R.warp = threadIdx.x >> 5;
  R.lane = threadIdx.x & 31;
  R.NG = FU_WARPS / G;
  R.g = R.warp / G;
  R.gt = G * 32;
  R.tg = threadIdx.x - R.g * R.gt;
  MfSmem<T> sm;
  {
    T* vs = reinterpret_cast<T*>(mf_smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(vs + R.NG * A.fmp);
    T* data = reinterpret_cast<T*>(full + R.NG * A.fNC);
    constexpr int RB = 16 / NK;
    for (int j = threadIdx.x; j < R.NG * A.fNC * RB * A.fmp; j += MT_THREADS) data[j] = T(0);  // read beyond the rows
    for (int j = threadIdx.x; j < R.NG * A.fNC; j += MT_THREADS) mbar_init(full + j, 1);
    fence_mbar_init();
    fence_proxy_async_smem();
    sm.vs = vs + R.g * A.fmp;
    sm.full = full + R.g * A.fNC;
    sm.kept = s_kept[R.g];
    sm.data = data + R.g * A.fNC * RB * A.fmp;
  }
  const int nworkers = gridDim.x * R.NG, wid = R.g * gridDim.x + blockIdx.x;
  int* abort_flag = A.ctl + 1;
  unsigned gen = 0;
  const T L2E = T(OTG_LOG2E);
  const T OUTF = LOGF ? T(OTG_LN2) : T(1);  // outputs: natural-log potentials or the scalings themselves
  for (int p = blockIdx.x; p < A.nprob; p += gridDim.x) {
    for (int i = threadIdx.x; i < A.rows[p]; i += MT_THREADS) {
      const int64_t ri = A.r_off[p] + i;
      if (LOGF) A.u[ri] = A.warm_u ? A.warm_u[ri] * L2E : T(0);
      else A.u[ri] = A.warm_u ? exp(A.warm_u[ri]) : T(1);
    }
    double mass = 0.0;
    if (LOGF) {
      for (int i = threadIdx.x; i < A.rows[p]; i += MT_THREADS) mass += widen(A.a[A.r_off[p] + i]);
      mass = block_sum_fixed(mass);
    }
    if (threadIdx.x == 0) {
      const int e = mass > 0.0 && isfinite(mass) ? ilogb(mass) + 1 : 0;
      A.flim[p] = sizeof(T) == 8 ? max(e - 985, -1000) : max(e - 70, -100);
      leaving[p] = 0;
      A.fbad[p] = 0;
      A.err2[p] = 0.0;
      if (A.and_depth > 0) A.and_cnt[p] = 0;
    }
  }
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < A.nprob; k += MT_THREADS) A.active[k] = k;
  if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) return;
  if (blockIdx.x == 0) mf_rebuild<T>(A, A.nprob, leaving, s_scan, nworkers);
  if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) return;

  T *vcur = A.v0, *vnxt = A.v1;
  MfRing ring{0, 0u, false};
  MfCursor<T> cur{};
  int nact = ld_acquire_i(A.ctl), na = ld_acquire_i(A.ctl + 7);
  bool ok = true;
  int ndec = 0;  // decisions taken (the same count in every CTA)
  auto look_up = [&]() {
    if (wid < na) {
      const MfShare S = mf_share(A, R, sm.kept, wid, na, nact);
      if (R.tg == 0) s_share[R.g] = S;
    }
    const MfPlace P = mf_first_place(A, na, nact);
    if (R.lane == 0) s_place[R.warp] = P;
    __syncthreads();
  };
  look_up();

  // the column update of the initial u: the first v
  if (wid < na) mf_colpass<T, LOGF, false>(A, R, wid, na, nact, (const T*)nullptr);
  if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) return;
  mf_merge<T, LOGF>(A, s_place[R.warp], na, nact, scr, (const T*)nullptr, vcur, [&](int, int64_t cj, T bj, T, T mx, T s, int) {
    vcur[cj] = LOGF ? lg2(bj) - lse_value(mx, s) : bj / s;
  });
  if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) return;

  for (int ii = 0;; ++ii) {
    // vcur: v of iteration ii, A.u: u of iteration ii - 1
    if (wid < na && !mf_pass<T, LOGF, NK>(A, R, sm, red, ring, cur, s_share[R.g], wid, nact, vcur)) ok = false;
    if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
    const bool check = ii % A.period == 0, last = ii + 1 == A.max_iter;
    int32_t* any_bad = A.leave_cnt + 2;
    if (blockIdx.x == 0 && threadIdx.x == 0) any_bad[(ii + 1) & 1] = 0;  // last read an iteration ago
    mf_merge<T, false>(A, s_place[R.warp], na, nact, scr, (const T*)nullptr, vcur, [&](int p, int64_t cj, T bj, T vo, T, T s, int lim) {
      if (check) {
        // column marginal of (u, v) of iteration ii, in the column's own slot
        const double cs = widen(LOGF ? s : vo * s) - widen(bj);
        A.e2col[cj] = cs * cs;
      }
      T vn;
      if (LOGF) {
        vn = bj == T(0) ? T(-INFINITY) : vo + lg2(bj / s);
        if (A.relax) vn = fma(A.omega, vn - vo, vo);
        if (bj != T(0) && !fu_at_least(s, exp2_of<T>(lim))) {  // terms may have underflowed
          vn = T(NAN);
          A.fbad[p] = 1;
          any_bad[ii & 1] = 1;
        }
      } else {
        vn = bj / s;
      }
      vnxt[cj] = vn;
    });
    if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
    const bool bad = LOGF && ld_acquire_i(any_bad + (ii & 1)) != 0;
    if (check || last) {
      bool joint_conv = false;
      if (A.joint && check) {
        // whole-batch stop: every problem's error, then the largest
        for (int k = blockIdx.x; k < nact; k += gridDim.x) {
          const int p = __ldcg(A.active + k);
          const double e2 = block_sum_slots(A.e2col + A.c_off[p], A.cols[p]);
          if (threadIdx.x == 0) A.err2[p] = e2;
        }
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        joint_conv = mt_joint_largest<T>(A, nact) < A.stop_thr;
      }
      int nleave = 0;
      for (int k = blockIdx.x; k < nact; k += gridDim.x) {
        const int p = __ldcg(A.active + k);
        double e = -1.0;
        bool conv = false;
        if (check) {
          // (one warp's square root: FP64 issues at two lanes per clock)
          const double e2 = A.joint ? __ldcg(A.err2 + p) : block_sum_slots(A.e2col + A.c_off[p], A.cols[p]);
          if (threadIdx.x == 0) e = sqrt(e2);
          conv = __syncthreads_or(threadIdx.x == 0 && (A.joint ? joint_conv : e < A.stop_thr));
        }
        const bool leave = conv || last;
        if (leave) {
          for (int i = threadIdx.x; i < A.rows[p]; i += MT_THREADS) A.out_u[A.r_off[p] + i] = __ldcg(A.u + A.r_off[p] + i) * OUTF;
          for (int j = threadIdx.x; j < A.cols[p]; j += MT_THREADS) A.out_v[A.c_off[p] + j] = __ldcg(vcur + A.c_off[p] + j) * OUTF;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          if (leave) {
            A.status[p] = conv ? OTG_STATUS_CONVERGED : OTG_STATUS_MAXITER;
            A.niter[p] = ii;
            A.err[p] = e;
          }
          leaving[p] = leave ? 1 : 0;
          nleave += leave ? 1 : 0;
        }
      }
      if (threadIdx.x == 0 && nleave) atomicAdd(A.leave_cnt + (ndec & 1), nleave);
      if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
      // the active list and its prefix sums change only when a problem left
      const bool changed = ld_acquire_i(A.leave_cnt + (ndec & 1)) != 0;
      if (blockIdx.x == 0 && threadIdx.x == 0) A.leave_cnt[(ndec + 1) & 1] = 0;  // last read a decision ago
      ++ndec;
      if (changed) {
        if (blockIdx.x == 0) mf_rebuild<T>(A, nact, leaving, s_scan, nworkers);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        nact = ld_acquire_i(A.ctl);
        na = ld_acquire_i(A.ctl + 7);
        if (nact == 0) break;
        // the shares are others now: what the ring has copied ahead is dropped
        if (ring.primed) {
          for (int q = 0; q < A.fNC; ++q) {
            if (!mbar_wait(sm.full + ring.slot, ring.phase, abort_flag, A.timeout_ns)) ok = false;
            if (++ring.slot == A.fNC) { ring.slot = 0; ring.phase ^= 1; }
          }
          mf_sync(R, G);
          ring.primed = false;
        }
        look_up();
      }
    }
    if (bad) {
      // column sums too small to trust (NaN in v): their update with running maxima
      if (wid < na) mf_colpass<T, LOGF, true>(A, R, wid, na, nact, vnxt);
      if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
      mf_merge<T, true>(A, s_place[R.warp], na, nact, scr, vnxt, vcur, [&](int, int64_t cj, T bj, T vo, T mx, T s, int) {
        const T vn = lg2(bj) - lse_value(mx, s);
        vnxt[cj] = A.relax ? fma(A.omega, vn - vo, vo) : vn;
      });
      if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
      for (int p = blockIdx.x * MT_THREADS + threadIdx.x; p < A.nprob; p += gridDim.x * MT_THREADS) A.fbad[p] = 0;
    }
    if ((check || last) && ld_acquire_i(A.ctl + 2)) {
      // handoff: the tail kernel continues with iteration ii + 1's row pass (its v is in vnxt)
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.ctl[3] = ii + 1;
        A.ctl[4] = vnxt == A.v1 ? 1 : 0;
        __threadfence();
        A.ctl[5] = 1;
      }
      break;
    }
    if constexpr (LOGF) {
      if (A.and_depth > 0) {
        mf_and_dots<T>(A, nact, vcur, vnxt);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        mf_and_solve<T>(A, nact);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
        mf_and_mix<T>(A, nact, vnxt);
        if (!fu_barrier(A.bar, gen, abort_flag, A.timeout_ns)) { ok = false; break; }
      }
    }
    { T* t = vcur; vcur = vnxt; vnxt = t; }
  }
  // copies in flight land before the CTA leaves
  if (ring.primed && R.tg == 0) {
    const uint64_t t0 = globaltimer();
    for (int q = 0; q < A.fNC; ++q) {
      while (!mbar_try_wait(sm.full + ring.slot, ring.phase)) if (globaltimer() - t0 > A.timeout_ns) break;
      if (++ring.slot == A.fNC) { ring.slot = 0; ring.phase ^= 1; }
    }
  }
  __syncthreads();
  (void)ok;
}

}  // namespace otg
