// The pipelined LU, one thread-block cluster per matrix: the kernels of one size class
// are one translation unit (kls_lu_64.cu and so on).  A module is loaded as a whole at
// the first call that needs a kernel of it, at about 0.5 ms a megabyte, and all classes
// together are 6.4 MB: the first determinant of a process 6.0 -> 1.8 ms.
#pragma once
#include "kls_lu_prims.cuh"
#include "kls_lu_pipe.h"
#include "kls_tcgen05.cuh"

namespace {

// ---- pipelined form: one thread-block cluster per matrix -----------------------
// Bound: the chain of N columns (pivot search, reciprocal, multipliers, update
// of the next column), not the flops.  So nothing but that chain is serial:
//  * every column belongs to one warp and lives in its registers (lane = row mod
//    32); no row is ever moved: each row carries its position in LAPACK's
//    order, and an exchange swaps two positions;
//  * the owner of column j + 1 updates it with column j's multipliers, factors
//    it and publishes it before it updates the rest of its columns, so the
//    warps run as a pipeline over the columns without a block or cluster
//    barrier: a column goes to a ring in the shared memory of every CTA of the
//    cluster and one mbarrier per slot announces it;
//  * 8 consecutive columns are on one CTA (kls_lu_cols.h), so most hand-overs stay
//    inside an SM.
// A slot is written again only when every warp has used it: each warp keeps a
// count of the columns it is done with, and the owner of every (slots / 2)-th
// column waits for all of them.
// Waits are bounded (KlsLuWait); one that runs out makes the determinant a NaN of its
// own, which the host turns into KLS_ERR_TIMEOUT.
//
// Measured (1 matrix, B200): N = 101 312 -> 97 us, 201 557 -> 267 us, 301 1022 ->
// 550 us against one CTA (101) or a cluster with one barrier per column; 16
// matrices 315 -> 99, 612 -> 348, 1990 -> 1097 us.  A column's chain is about
// 1600 cycles at 4 rows a lane and 3300 at 10 (hand-over 160 / 360, update 280 / 540,
// pivot search with its reciprocal 670 / 1260, broadcast 60 / 80, multipliers and
// publication 440 / 1100; the marks themselves are some 50 each): about 350
// instructions that depend on one another.

__device__ __forceinline__ void st_cluster_v2(uint32_t addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y)
               : "memory");
}
__device__ __forceinline__ void st_cluster_v2i(uint32_t addr, int a, int b) {
  asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr)
               : "memory");
}
__device__ __forceinline__ int ld_acquire_cluster(uint32_t addr) {
  int v;
  asm volatile("ld.acquire.cluster.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_cluster(uint32_t addr, int v) {
  asm volatile("st.release.cluster.shared::cta.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Bounded wait.  The waiting warp is suspended (up to 10 us a try) instead of
// polling: seven polling warps slow the one that the others wait for (its
// shuffles and shared-memory reads queue behind theirs).  Only the warp whose
// column is next polls for a while, as it wakes up the sooner (N = 301 576 -> 556
// us, 16 matrices of 201 374 -> 352).
__device__ __forceinline__ bool lup_wait(uint32_t bar, uint32_t parity, volatile int* abort,
                                         bool poll, unsigned long long limit) {
  for (int it = 0; poll && it < 200; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 10000;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*abort) return false;
    if ((it & 15) == 15) {
      const unsigned long long t = kls_tc::globaltimer();
      if (!t0) t0 = t;
      else if (t - t0 > limit) {
        *abort = 1;
        return false;
      }
    }
  }
}

// element `row` (warp-uniform) of a column held as lane = row & 31, a[row >> 5]
template <int RPL>
__device__ __forceinline__ double2 lup_row(const double2 (&a)[RPL], int row) {
  double2 v = a[0];
  const int q = row >> 5;
#pragma unroll
  for (int r = 1; r < RPL; ++r)
    if (q == r) v = a[r];
  return make_double2(__shfl_sync(0xffffffffu, v.x, row & 31),
                      __shfl_sync(0xffffffffu, v.y, row & 31));
}

// RPL rows per lane, LP columns per warp
template <int RPL, int LP>
__device__ __forceinline__ void lup_body(int n, int slots, const double2* __restrict__ A,
                                         double2* __restrict__ det, double* __restrict__ logabs,
                                         unsigned char* smem, const KlsLuWait& wait) {
  using namespace kls_tc;
  __shared__ int prog[LUP_WARPS];             // columns each warp is done with
  __shared__ volatile int s_abort;
  __shared__ int s_failed;                    // rank 0: a wait ran out somewhere
  uint32_t rank, C;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* ring = reinterpret_cast<double2*>(smem);                 // [slots][n]
  LupMeta* meta = reinterpret_cast<LupMeta*>(ring + (size_t)slots * n);
  uint64_t* full = reinterpret_cast<uint64_t*>(meta + slots);
  if (tid < LUP_WARPS) prog[tid] = 0;
  if (tid == 0) { s_abort = 0; s_failed = 0; }
  for (int s = tid; s < slots; s += LUP_THREADS) mbar_init(smem_u32(full + s), 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  LupCols own(n, (int)C, (int)rank, warp, LP);
  double2 a[LP][RPL];
  int pos[RPL];
#pragma unroll
  for (int r = 0; r < RPL; ++r) {
    const int i = lane + 32 * r;
    pos[r] = i < n ? i : -1;
#pragma unroll
    for (int lp = 0; lp < LP; ++lp) {
      const int g = own.col(lp);
      a[lp][r] = make_double2(0.0, 0.0);
      if (i < n && g < n) KLS_IF(LU_IN(i, g)) a[lp][r] = A[(size_t)i * n + g];
    }
  }
  cluster_sync_all();                         // barriers initialised everywhere

  // pivot search, multipliers and publication (slot s) of local column c = global g
  auto factor = [&](double2 (&c)[RPL], int g, int s) {
    // a lane's largest |re| + |im| by its upper 32 bits, and that entry's
    // reciprocal, which runs while the warp looks for the largest of all
    unsigned hm = 0;
    double2 best = make_double2(1.0, 0.0);
    unsigned at = 0;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const double m = fabs(c[r].x) + fabs(c[r].y);
      const unsigned h = pos[r] >= g && m == m ? (unsigned)__double2hiint(m) | 0x80000000u : 0u;
      if (h > hm) {
        hm = h;
        best = c[r];
        at = ((unsigned)pos[r] << 16) | (unsigned)(lane + 32 * r);
      }
    }
    double2 rb = cinv(best.x, best.y);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hm);
    int ties = 0;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const double m = fabs(c[r].x) + fabs(c[r].y);
      if (pos[r] >= g && m == m && ((unsigned)__double2hiint(m) | 0x80000000u) == mh) ++ties;
    }
    const unsigned who = __ballot_sync(0xffffffffu, ties > 0);
    const unsigned more = __ballot_sync(0xffffffffu, ties > 1);
    int src = __ffs(who) - 1;
    if (mh == 0u || more || (who & (who - 1))) {
      // several entries with these bits: all 64 of them, then the position; no
      // comparable entry at all: the diagonal
      unsigned lm = 0;
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const double m = fabs(c[r].x) + fabs(c[r].y);
        if (mh && pos[r] >= g && m == m && ((unsigned)__double2hiint(m) | 0x80000000u) == mh)
          lm = max(lm, (unsigned)__double2loint(m));
      }
      lm = __reduce_max_sync(0xffffffffu, lm);
      unsigned cand = 0xffffffffu;
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const double m = fabs(c[r].x) + fabs(c[r].y);
        const bool in = mh ? pos[r] >= g && m == m &&
                                 ((unsigned)__double2hiint(m) | 0x80000000u) == mh &&
                                 (unsigned)__double2loint(m) == lm
                           : pos[r] == g;
        const unsigned x = ((unsigned)pos[r] << 16) | (unsigned)(lane + 32 * r);
        if (in && x < cand) { cand = x; best = c[r]; }
      }
      at = __reduce_min_sync(0xffffffffu, cand);
      src = (int)(at & 31u);
      rb = cinv(best.x, best.y);
    }
    at = __shfl_sync(0xffffffffu, at, src);
    const int piv = (int)(at & 0xffffu), q = (int)(at >> 16);
    const double2 u = make_double2(__shfl_sync(0xffffffffu, best.x, src),
                                   __shfl_sync(0xffffffffu, best.y, src));
    double2 ru = make_double2(__shfl_sync(0xffffffffu, rb.x, src),
                              __shfl_sync(0xffffffffu, rb.y, src));
    if (u.x == 0.0 && u.y == 0.0) ru = make_double2(0.0, 0.0);
    if (slots < n && g >= slots && g % (slots / 2) == 0) {
      // every warp of the cluster is done with the columns whose slots the
      // next slots / 2 columns take
      const int need = g - slots + slots / 2;
      for (int w = lane; w < (int)C * LUP_WARPS; w += 32) {
        const uint32_t ad = mapa_u32(smem_u32(&prog[w % LUP_WARPS]), w / LUP_WARPS);
        unsigned long long t0 = 0;
        for (uint32_t it = 0; ld_acquire_cluster(ad) < need; ++it) {
          if (s_abort) break;
          if ((it & 63) == 63) {
            const unsigned long long t = globaltimer();
            if (!t0) t0 = t;
            else if (t - t0 > wait.ns) { s_abort = 1; break; }
          }
        }
      }
      __syncwarp();
    }
    double2* slot = ring + (size_t)s * n;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      if (i < n)
        slot[i] = pos[r] >= g && i != piv ? cmul(c[r], ru) : make_double2(0.0, 0.0);
    }
    if (lane == 0) { meta[s].u = u; meta[s].piv = piv; meta[s].pos = q; }
    __syncwarp();
    if (lane == 0 && g != wait.skip) mbar_arrive(smem_u32(full + s));
    // the other CTAs, the next one first.  One CTA at a time: the release waits
    // for its stores, so the SM's path to the cluster never fills up with
    // stores that the other warps' shared-memory accesses would queue behind.
    for (uint32_t t = 1; t < C; ++t) {
      const uint32_t to = rank + t < C ? rank + t : rank + t - C;
      const uint32_t base = mapa_u32(smem_u32(slot), to);
#pragma unroll
      for (int r = 0; r < RPL; ++r)            // (this lane's own values, read back)
        if (lane + 32 * r < n) st_cluster_v2(base + (lane + 32 * r) * 16, slot[lane + 32 * r]);
      if (lane == 0) {
        const uint32_t mb = mapa_u32(smem_u32(meta + s), to);
        st_cluster_v2(mb, u);
        st_cluster_v2i(mb + 16, piv, q);
      }
      __syncwarp();
      if (lane == 0 && g != wait.skip) arrive_cluster(mapa_u32(smem_u32(full + s), to));
    }
  };

  const bool keeper = rank == 0 && warp == 0;  // multiplies the pivots up, in order
  LuDet acc;
  // a[0] is the warp's next column (index own.next), a[1 .. left - 1] those after it
  auto shift = [&]() {
#pragma unroll
    for (int lp = 0; lp + 1 < LP; ++lp)
#pragma unroll
      for (int r = 0; r < RPL; ++r) a[lp][r] = a[lp + 1][r];
    own.taken();
  };
  if (own.next == 0) {
    factor(a[0], 0, 0);
    shift();
  }
  const int until = keeper ? n : own.last;     // columns this warp has to take in
  int j = 0, s = 0;                            // column j is in slot s
  uint32_t parity = 0;
  for (; j < until; ++j) {
    const bool ok = lup_wait(smem_u32(full + s), parity, &s_abort,
                             own.next == j + 1 || j + 1 == until, wait.ns);
    if (!__all_sync(0xffffffffu, ok)) break;
    const LupMeta mt = meta[s];
#pragma unroll
    for (int r = 0; r < RPL; ++r) {            // the exchange of positions j and mt.pos
      const bool here = lane + 32 * r == mt.piv;
      pos[r] = here ? j : pos[r] == j ? mt.pos : pos[r];
    }
    const double2* slot = ring + (size_t)s * n;
    if (own.next == j + 1) {                   // the chain: this column is wanted next
      const double2 u = lup_row<RPL>(a[0], mt.piv);
#pragma unroll
      for (int r = 0; r < RPL; ++r)
        if (lane + 32 * r < n) a[0][r] = lu_update(a[0][r], slot[lane + 32 * r], u);
      factor(a[0], own.next, s + 1 < slots ? s + 1 : 0);
      shift();
    }
    if (own.left) {
      double2 u[LP];
#pragma unroll
      for (int lp = 0; lp < LP; ++lp)
        if (lp < own.left) u[lp] = lup_row<RPL>(a[lp], mt.piv);
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        if (lane + 32 * r >= n) continue;
        const double2 l = slot[lane + 32 * r];
#pragma unroll
        for (int lp = 0; lp < LP; ++lp)
          if (lp < own.left) a[lp][r] = lu_update(a[lp][r], l, u[lp]);
      }
    }
    if (keeper) acc.times(mt.u, mt.pos != j);
    if (slots < n) {
      __syncwarp();
      if (lane == 0 && (j & 3) == 3) st_release_cluster(smem_u32(&prog[warp]), j + 1);
    }
    if (++s == slots) { s = 0; parity ^= 1u; }
  }
  __syncwarp();
  if (lane == 0) {
    st_release_cluster(smem_u32(&prog[warp]), n);
    if (j < until || s_abort) {                // a wait ran out
      const uint32_t f = mapa_u32(smem_u32(&s_failed), 0);
      asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(f), "r"(1) : "memory");
    }
  }
  __syncwarp();
  cluster_sync_all();                          // nobody leaves while others write here
  if (keeper && lane == 0) {
    if (s_failed) {
      const double x = __longlong_as_double((long long)KLS_NAN_LU_TIMEOUT);
      *det = make_double2(x, x);
      if (logabs) *logabs = x;
    } else {
      acc.store(det, logabs);
    }
  }
}

template <int RPL, int LP>
__global__ void __launch_bounds__(LUP_THREADS)
lu_pipe_kernel(int n, int slots, int C, const double2* __restrict__ Aall,
               double2* __restrict__ det_out, double* __restrict__ logabs_out,
               const __grid_constant__ KlsLuWait wait) {
  extern __shared__ __align__(16) unsigned char lsm[];
  const int m = blockIdx.x / C;
  lup_body<RPL, LP>(n, slots, Aall + (size_t)m * n * n, det_out + m,
                    logabs_out ? logabs_out + m : nullptr, lsm, wait);
}

// one (model, omega) pair per cluster; the ring holds `smem` bytes
template <int RPL, int LP>
__global__ void __launch_bounds__(LUP_THREADS)
multi_lu_pipe_kernel(const kls_mdesc* __restrict__ md, const int2* __restrict__ pairs, int C,
                     int max_slots, const __grid_constant__ KlsLuWait wait) {
  extern __shared__ __align__(16) unsigned char lsm[];
  const int2 pz = pairs[blockIdx.x / C];
  const kls_mdesc& d = md[pz.x];
  lup_body<RPL, LP>(d.Na, d.Na < max_slots ? d.Na : max_slots, d.A + (size_t)pz.y * d.Na * d.Na,
                    d.det + pz.y, d.logabs + pz.y, lsm, wait);
}

}  // namespace

// the kernels of the class up to n rows: RPL rows per lane, LP columns per warp
#define LUP_DEFINE(n, RPL, LP, WIDE)                                                          \
  LupKernels lup_kernels_##n() {                                                              \
    return {(const void*)lu_pipe_kernel<RPL, LP>, (const void*)multi_lu_pipe_kernel<RPL, LP>, \
            WIDE};                                                                            \
  }
