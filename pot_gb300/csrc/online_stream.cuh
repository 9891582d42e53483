// Shifted-sum pass of the online log-Sinkhorn (one problem, d <= 64), two
// CTAs sharing every streamed tile.
//
// What bounds it: 13 MMAs of 128 x 128 x 16 per 128 x 128 pairs (832 tensor
// cycles; the exponentials take 512).  With one row block per CTA and
// 128-point tiles every CTA read 36 KiB per tile from L2 at 22 B per
// SM-cycle: 1660 cycles a tile, and n = 16384 left 24 of 152 SMs without a
// row block.  Here
//   - a cluster of two CTAs owns two row blocks and takes them as one M = 256
//     MMA (cta_group::2): each CTA holds its own row block and one half of
//     the 256-point tile, both loaded for itself alone (18 KiB per 128 points
//     and SM), the MMA reads the halves of both, and each CTA's TMEM gets its
//     own 128 rows;
//   - N = 256: per 128 cycles a CTA reads 8 KiB of shared memory, where two
//     N = 128 MMAs of one CTA read 16 KiB, all that the shared memory
//     delivers, with the arriving tiles still to be written;
//   - the (row pair, tile) units are cut into one contiguous range per
//     cluster; a row pair that several clusters share leaves its row sums in
//     slots, and the last CTA to arrive adds the slots in order (the sums are
//     all relative to the row's one shift) and finishes the rows.  No CTA
//     waits for another cluster.
// Measured, a pass and its fix-up (time of 30 more iterations over 60): 16384
// x 16384, d = 64: 62.3 us, 19456 x 19456: 79.8, 65536 x 65536: 936; with the
// halves copied into both CTAs and an N = 256 MMA in each: 64.3, 84.2, 979.
// (With a row block per CTA and 128-point tiles the pass alone took 106.6 at
// 16384 x 16384.)  3000 x 3000, d = 40: 12.8; 500 x 500, d = 10 (launch
// latency): 8.8.  Programmatic
// launches of the pass and of its fix-up: 30 iterations at 16384 x 16384 4.63
// -> 4.40 ms, at 500 x 500 1.05 -> 0.82 ms.
// Stages hold one plane of a CTA's half tile (hi, then lo with the extension
// columns) so that a stage is free after 8 or 5 MMAs; two resident row tiles,
// two 256-column accumulators.
//
// Barriers of the pair.  The even CTA (the leader) issues the MMAs, so its
// barriers count what both CTAs load (`full`, `res_full`: each CTA's copies
// complete on the leader's barrier) and what both epilogues release (`acce`).
// The MMAs' completion arrives in both (`empty`, `res_empty`, `accf`).
#pragma once

namespace otg {

constexpr int OS_N = 256;              // streamed points per tile
constexpr int OS_NBUF = 2;             // TMEM accumulators of 256 columns
constexpr int OS_MAXST = 16;           // barrier slots (stages): 8 wide, 16 narrow
constexpr int OS_MAX_CLUSTERS = 128;   // ranges of a pass at most (room for their partial sums)

// Shared-memory plan by plane width (64 or 16 halves).
template <bool NARROW> struct OsGeo {
  static constexpr uint32_t row = NARROW ? 32 : 128;           // bytes of a plane row
  static constexpr uint32_t plane = OL_M * row;                // a stage: one plane of half a tile
  static constexpr int ns = NARROW ? 16 : 8;                   // stages
  static constexpr uint32_t res = 2 * plane + OL_EXT;          // resident hi, lo, extension
  static constexpr uint32_t ring = ns * plane, ext = ns / 2 * OL_EXT;
  static constexpr uint32_t bytes = 2 * res + ring + ext;
};
static_assert(OsGeo<false>::res % 1024 == 0 && OsGeo<true>::res % 1024 == 0, "swizzle atoms stay aligned");
constexpr size_t OS_SMEM_EXTRA = 1024 /*align*/ + 512 /*barriers, flags*/ + 3 * OL_M * 4 /*column groups' sums*/;

struct OsWork {          // what a pass adds to OnlinePass
  int row_pairs, tiles;  // pairs of row blocks, 256-point tiles
  int clusters;          // ranges: gridDim.x / 2
  float* part;           // partial row sums: slot s of row pair p at (base(p) + s) * 256
  unsigned* cnt;         // [2 * row_pairs] arrivals (zero between passes)
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared::cluster address of an object of the leader at this CTA's offset.
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_addr(p)));
  return r;
}
// TMA load into this CTA whose bytes complete on the leader's barrier.
__device__ __forceinline__ void tma_load_2d_leader(void* dst, const CUtensorMap* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      :: "r"(smem_addr(dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// Arrive on the leader's barrier.  (Nothing in memory is handed over, only
// TMEM columns, which the tcgen05 fences order: no cluster-scope release,
// whose fence cost 0.27 us a tile: 16384 x 16384, d = 64, 77 us a pass.)
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" :: "r"(bar) : "memory");
}
// D (+)= A B^T over the pair: rows of both CTAs' A tiles, points of both
// halves of B (descriptors: the same offsets in either CTA).  Leader only.
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs of the pair once every
// MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      :: "r"(smem_addr(bar)), "h"((unsigned short)3) : "memory");
}
// TMEM of the pair, by one full warp of each CTA.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(slot)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(ncols) : "memory");
}

// Programmatic launches (a no-op in ordinary ones): the next kernel may be
// set up from now on; wait for the kernel before to end.
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The range of units [first, last) of cluster c, and the cluster of unit u.
__host__ __device__ __forceinline__ int64_t os_first(int64_t c, int64_t units, int64_t clusters) {
  return c * units / clusters;
}
__host__ __device__ __forceinline__ int64_t os_owner(int64_t u, int64_t units, int64_t clusters) {
  return ((u + 1) * clusters - 1) / units;
}

template <bool NARROW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(OL_THREADS, 1)
online_stream_kernel(const __grid_constant__ CUtensorMap tAh, const __grid_constant__ CUtensorMap tAl,
                     const __grid_constant__ CUtensorMap tBh, const __grid_constant__ CUtensorMap tBl,
                     const __grid_constant__ CUtensorMap tR, const __grid_constant__ CUtensorMap tS, OnlinePass P,
                     OsWork W) {
  using G = OsGeo<NARROW>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* resident = smem;                       // two slots
  unsigned char* ring = smem + 2 * G::res;
  unsigned char* exts = ring + G::ring;
  uint64_t* bars = reinterpret_cast<uint64_t*>(exts + G::ext);
  uint64_t* res_full = bars;                            // [2]
  uint64_t* res_empty = bars + 2;                       // [2]
  uint64_t* accf = bars + 4;                            // [OS_NBUF]
  uint64_t* acce = bars + 6;                            // [OS_NBUF]
  uint64_t* full = bars + 8;                            // [OS_MAXST]
  uint64_t* empty = full + OS_MAXST;                    // [OS_MAXST]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(empty + OS_MAXST);
  int* uflag = reinterpret_cast<int*>(tslot + 1);       // a row of the unit failed
  int* dead = uflag + 1;                                // an epilogue warp gave up
  int* last = uflag + 2;                                // this CTA finishes the row block
  float* red = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(bars) + 512);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank(), cid = blockIdx.x >> 1;
  const int T = W.tiles;
  const int64_t units = (int64_t)W.row_pairs * T;
  const int64_t u0 = os_first(cid, units, W.clusters), u1 = os_first(cid + 1, units, W.clusters);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 2; ++k) { mbar_init(res_full + k, 1); mbar_init(res_empty + k, 1); }
    for (int k = 0; k < OS_NBUF; ++k) { mbar_init(accf + k, 1); mbar_init(acce + k, 2 * OL_EPI); }
    for (int k = 0; k < OS_MAXST; ++k) { mbar_init(full + k, 1); mbar_init(empty + k, 1); }
    *uflag = 0;
    *dead = 0;
    fence_mbar_init();
    prefetch_tmap(&tAh); prefetch_tmap(&tAl); prefetch_tmap(&tBh); prefetch_tmap(&tBl); prefetch_tmap(&tR); prefetch_tmap(&tS);
  }
  if (warp == OL_EPI + 1) tmem_alloc_pair(tslot, OS_NBUF * OS_N);
  tc_fence_before();
  cluster_sync_all();  // the peer's barriers are set before anything arrives on them
  tc_fence_after();
  grid_launch_next();
  grid_wait_before();  // nothing above reads what the kernel before wrote
  const uint32_t tmem = *tslot;

  if (warp == OL_EPI) {
    // producer: per segment (row pair, tiles of the range) the CTA's own
    // resident rows, then its half of every tile; the leader's barriers
    // expect both CTAs' bytes
    if (lane == 0) {
      const bool leader = rank == 0;
      int q = 0, seg = 0;
      bool ok = true;
      for (int64_t u = u0; u < u1 && ok; ++seg) {
        const int rp = (int)(u / T), t0 = (int)(u % T), t1 = (int)(u1 - u < T - t0 ? t0 + (u1 - u) : T);
        const int r0 = (2 * rp + rank) * OL_M, rs = seg & 1;
        if (seg > 1 && !mbar_wait(res_empty + rs, ((seg >> 1) - 1) & 1, P.abort_flag, P.timeout_ns)) { ok = false; break; }
        unsigned char* res = resident + rs * G::res;
        const uint32_t rbar = leader_addr(res_full + rs);
        if (leader) mbar_arrive_expect_tx(res_full + rs, 2 * G::res);
        tma_load_2d_leader(res, &tAh, 0, r0, rbar);
        tma_load_2d_leader(res + G::plane, &tAl, 0, r0, rbar);
        tma_load_2d_leader(res + 2 * G::plane, &tR, 0, r0, rbar);
        for (int k = 0; k < 2 * (t1 - t0); ++k, ++q) {
          const int s = q % G::ns, y = (t0 + (k >> 1)) * OS_N + rank * OL_M;
          if (!mbar_wait(empty + s, ((q / G::ns) & 1) ^ 1, P.abort_flag, P.timeout_ns)) { ok = false; break; }
          const uint32_t bar = leader_addr(full + s);
          if (leader) mbar_arrive_expect_tx(full + s, 2 * (G::plane + ((k & 1) ? OL_EXT : 0u)));
          tma_load_2d_leader(ring + s * G::plane, (k & 1) ? &tBl : &tBh, 0, y, bar);
          if (k & 1) tma_load_2d_leader(exts + (s >> 1) * OL_EXT, &tS, 0, y, bar);
        }
        u += t1 - t0;
      }
      // Copies in flight land and the MMAs' arrivals are in before the CTA
      // leaves (the leader's waits cover the copies of both; the pair leaves
      // together).
      const uint64_t w0 = globaltimer();
      for (int k = q > G::ns ? q - G::ns : 0; k < q; ++k) {
        if (leader)
          while (!mbar_try_wait(full + k % G::ns, (k / G::ns) & 1)) if (globaltimer() - w0 > P.timeout_ns) break;
        while (!mbar_try_wait(empty + k % G::ns, (k / G::ns) & 1)) if (globaltimer() - w0 > P.timeout_ns) break;
      }
      for (int k = seg > 2 ? seg - 2 : 0; k < seg; ++k) {
        if (leader)
          while (!mbar_try_wait(res_full + (k & 1), (k >> 1) & 1)) if (globaltimer() - w0 > P.timeout_ns) break;
        while (!mbar_try_wait(res_empty + (k & 1), (k >> 1) & 1)) if (globaltimer() - w0 > P.timeout_ns) break;
      }
    }
  } else if (warp == OL_EPI + 1) {
    // MMA issuer
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = umma_idesc_f16(2 * OL_M, OS_N, false);
      int q = 0, n = 0, seg = 0;
      bool ok = true;
      for (int64_t u = u0; u < u1 && ok; ++seg) {
        const int t0 = (int)(u % T), t1 = (int)(u1 - u < T - t0 ? t0 + (u1 - u) : T), rs = seg & 1;
        const unsigned char* res = resident + rs * G::res;
        if (!mbar_wait(res_full + rs, (seg >> 1) & 1, P.abort_flag, P.timeout_ns)) break;
        for (int t = t0; t < t1; ++t, ++n) {
          const int b = n % OS_NBUF;
          if (!mbar_wait(acce + b, ((n / OS_NBUF) & 1) ^ 1, P.abort_flag, P.timeout_ns)) { ok = false; break; }
          const uint32_t dst = tmem + (uint32_t)(b * OS_N);
          const uint64_t ah = NARROW ? umma_desc_k32(res) : umma_desc_k128(res);
          const uint64_t al = NARROW ? umma_desc_k32(res + G::plane) : umma_desc_k128(res + G::plane);
          int s = q % G::ns;
          if (!mbar_wait(full + s, (q / G::ns) & 1, P.abort_flag, P.timeout_ns)) { ok = false; break; }
          tc_fence_after();
          const uint64_t bh = NARROW ? umma_desc_k32(ring + s * G::plane) : umma_desc_k128(ring + s * G::plane);
#pragma unroll
          for (int kk = 0; kk < (NARROW ? 1 : OL_K / 16); ++kk) {
            const uint64_t o = (uint64_t)(kk * 32) >> 4;
            umma_f16_pair(dst, ah + o, bh + o, idesc, kk ? 1u : 0u);
            umma_f16_pair(dst, al + o, bh + o, idesc, 1);
          }
          umma_commit_pair(empty + s);
          ++q;
          s = q % G::ns;
          if (!mbar_wait(full + s, (q / G::ns) & 1, P.abort_flag, P.timeout_ns)) { ok = false; break; }
          tc_fence_after();
          const uint64_t bl = NARROW ? umma_desc_k32(ring + s * G::plane) : umma_desc_k128(ring + s * G::plane);
#pragma unroll
          for (int kk = 0; kk < (NARROW ? 1 : OL_K / 16); ++kk) {
            const uint64_t o = (uint64_t)(kk * 32) >> 4;
            umma_f16_pair(dst, ah + o, bl + o, idesc, 1);
          }
          umma_f16_pair(dst, umma_desc_k32(res + 2 * G::plane), umma_desc_k32(exts + (s >> 1) * OL_EXT), idesc, 1);
          umma_commit_pair(empty + s);
          ++q;
          umma_commit_pair(accf + b);
        }
        if (ok) umma_commit_pair(res_empty + rs);
        u += t1 - t0;
      }
      // every MMA has completed before the accumulators go
      const uint64_t w0 = globaltimer();
      for (int k = n > OS_NBUF ? n - OS_NBUF : 0; k < n; ++k)
        while (!mbar_try_wait(accf + k % OS_NBUF, (k / OS_NBUF) & 1)) if (globaltimer() - w0 > P.timeout_ns) break;
    }
  } else {
    // epilogue: warp w reads TMEM lane quarter w % 4 (rows 32 (w % 4) + lane)
    // and columns 64 (w / 4) .. +63 of each tile
    const int quarter = warp & 3, cgrp = warp >> 2;
    const int row_local = quarter * 32 + lane;
    int n = 0;
    for (int64_t u = u0; u < u1;) {
      const int rp = (int)(u / T), t0 = (int)(u % T), t1 = (int)(u1 - u < T - t0 ? t0 + (u1 - u) : T);
      const int rb = 2 * rp + rank, row = rb * OL_M + row_local;
      const OlRowIn rin = ol_row_in<OL_FSUM>(P, row, cgrp == 0 && row < P.n_rows);
      float sm = 0.f, sc = 0.f;
      int ok = 1;
      for (int t = t0; t < t1; ++t, ++n) {
        const int b = n % OS_NBUF;
        if (lane == 0) ok = mbar_wait(accf + b, (n / OS_NBUF) & 1, P.abort_flag, P.timeout_ns) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        if (!ok) break;
        tc_fence_after();
        const uint32_t addr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * OS_N + cgrp * 64);
        uint32_t v[32];
        tmem_ld32u(addr, v);
        ol_fsum_acc(v, sm, sc);
        tmem_ld32u(addr + 32, v);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(leader_addr(acce + b));
        ol_fsum_acc(v, sm, sc);
      }
      if (!ok) *dead = 1;
      if (cgrp > 0) red[(cgrp - 1) * OL_M + row_local] = sm;
      named_bar(1, OL_EPI * 32);
      if (*dead) break;  // the same for every epilogue warp
      const bool whole = t1 - t0 == T;
      bool done = true;
      if (cgrp == 0) {
        for (int g = 0; g < 3; ++g) sm += red[g * OL_M + row_local];
        if (!whole) {
          // row pair rp: owners c0 .. c1, slot of the range = its number from c0;
          // slots of earlier pairs: at most one per range begun plus one per pair
          const int64_t c0 = os_owner((int64_t)rp * T, units, W.clusters);
          const int64_t c1 = os_owner((int64_t)(rp + 1) * T - 1, units, W.clusters);
          float* slots = W.part + (c0 + rp) * OS_N + rank * OL_M + row_local;
          __stcg(slots + (cid - c0) * OS_N, sm);
          __threadfence();
          named_bar(2, OL_M);
          if (threadIdx.x == 0) {
            const unsigned was = atomicAdd(W.cnt + rb, 1u);
            const int fin = was == (unsigned)(c1 - c0);
            if (fin) W.cnt[rb] = 0u;
            __threadfence();
            *last = fin;
          }
          named_bar(2, OL_M);
          done = *last != 0;
          if (done) {
            sm = 0.f;
            const int ns = (int)(c1 - c0) + 1;
            for (int k = 0; k < ns; k += 8) {
              float p[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) p[j] = k + j < ns ? __ldcg(slots + (int64_t)(k + j) * OS_N) : 0.f;
#pragma unroll
              for (int j = 0; j < 8; ++j) sm += p[j];
            }
          }
        }
        if (done && !ol_row_finish<OL_FSUM>(P, row, row, 0.f, sm, rin)) *uflag = 1;
      }
      // the groups' sums are read, and the failures marked, before the next segment
      named_bar(1, OL_EPI * 32);
      if (threadIdx.x == 0) ol_note_unit(P, uflag, 0, rb * OL_M);
      u += t1 - t0;
    }
  }
  tc_fence_before();
  cluster_sync_all();  // nothing of the pair's is in flight towards either CTA
  if (warp == OL_EPI + 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, OS_NBUF * OS_N);
  }
}

}  // namespace otg
