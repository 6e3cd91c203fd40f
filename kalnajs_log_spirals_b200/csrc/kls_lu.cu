// det(I - M(omega)) for a batch of matrices: complex FP64 LU with partial
// pivoting (the reference moves M to the host and calls LinearAlgebra.det ->
// LAPACK zgetrf, MatrixBuilder.jl:173-182).
//
// Pivot choice follows LAPACK's izamax (largest |re| + |im|, first index on
// ties); the column is scaled by the reciprocal of the pivot as zgetf2 does.
// The determinant is accumulated as a mantissa and a binary exponent so that
// products of ~N_alpha pivots neither overflow nor underflow; the result is
// returned both as a complex number and as log|det|.
//
// lu_pipe_kernel (N <= 512): one thread-block cluster per matrix, the matrix in
// registers, columns passed from warp to warp; lu_det_kernel: one CTA per
// matrix through L2, any N, and batches of many matrices (lup_wins, kls_lu_cols.h).
// Both return the same bits.
#include "kls_internal.cuh"
#include "kls_lu_cols.h"
#include "kls_tcgen05.cuh"
#include <algorithm>
#include <cfloat>

namespace {

constexpr int LU_THREADS = 1024;

// 1/(c + i d) = (c - i d) / (c^2 + d^2) on values scaled by a power of two (one
// reciprocal on the factorisation's serial chain); Smith's two divisions where
// the exponent leaves no room to scale
__device__ __forceinline__ double2 cinv(double c, double d) {
  const int ex = max(__double2hiint(c) & 0x7ff00000, __double2hiint(d) & 0x7ff00000);
  if (ex > (64 << 20) && ex < (1982 << 20)) {
    const double s = __hiloint2double(0x7fe00000 - ex, 0);
    const double x = __dmul_rn(c, s), y = __dmul_rn(d, s);
    const double t = __dmul_rn(__drcp_rn(__fma_rn(x, x, __dmul_rn(y, y))), s);
    return make_double2(__dmul_rn(x, t), __dmul_rn(-y, t));
  }
  if (fabs(d) <= fabs(c)) {
    double r = d / c, t = 1.0 / (c + d * r);
    return make_double2(t, -r * t);
  }
  double r = c / d, t = 1.0 / (d + c * r);
  return make_double2(r * t, -t);
}

// roundings pinned (no compiler choice of which product joins an FMA), so
// every kernel that inlines the LU body gives the same bits
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)),
                      __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}

// a - l p
__device__ __forceinline__ double2 lu_update(double2 a, double2 l, double2 p) {
  return make_double2(__fma_rn(l.y, p.y, __fma_rn(-l.x, p.x, a.x)),
                      __fma_rn(-l.y, p.x, __fma_rn(-l.x, p.y, a.y)));
}

// running determinant: mant * 2^expo
struct LuDet {
  double2 mant = make_double2(1.0, 0.0);
  long long expo = 0;
  bool zero = false;
  __device__ __forceinline__ void normalise() {
    const double mx = fmax(fabs(mant.x), fabs(mant.y));
    if (mx != 0.0 && isfinite(mx)) {
      const int e = ilogb(mx);
      mant.x = scalbn(mant.x, -e);
      mant.y = scalbn(mant.y, -e);
      expo += e;
    }
  }
  // scaling by powers of two is exact, so it is done only when it is needed
  __device__ __forceinline__ void times(double2 u, bool swapped) {
    if (swapped) { mant.x = -mant.x; mant.y = -mant.y; }
    if (u.x == 0.0 && u.y == 0.0) zero = true;
    mant = cmul(mant, u);
    const double mx = fmax(fabs(mant.x), fabs(mant.y));
    if (!(mx > 0x1p-100 && mx < 0x1p100)) normalise();
  }
  __device__ __forceinline__ void store(double2* det, double* logabs) {
    normalise();
    double2 d = make_double2(0.0, 0.0);
    double la = -INFINITY;
    if (!zero) {
      const long long e = expo > 4000 ? 4000 : expo < -4000 ? -4000 : expo;
      d = make_double2(scalbn(mant.x, (int)e), scalbn(mant.y, (int)e));
      la = log(hypot(mant.x, mant.y)) + (double)expo * 0.69314718055994530942;
    }
    *det = d;
    if (logabs) *logabs = la;
  }
};

// element (i, c) of the n x n matrix A, guarded in the bounds-checked build
#define LU_IN(i, c) KLS_IB((int64_t)(i) * n + (c), (int64_t)n * n, KS_LU)
#define LU_A(i, c) KLS_LD(LU_IN(i, c), A[(size_t)i * n + c], make_double2(0.0, 0.0))

// LU of one n x n row-major matrix A by the whole CTA; writes *det_out and,
// if given, *logabs_out.  sh holds 2 n complex values.
__device__ __forceinline__ void lu_det_body(int n, double2* __restrict__ A, double2* sh,
                                            double2* __restrict__ det_out,
                                            double* __restrict__ logabs_out) {
  double2* prow = sh;
  double2* lcol = sh + n;
  __shared__ double red_v[32];
  __shared__ int red_i[32];
  __shared__ int s_piv;
  __shared__ double2 s_u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;

  LuDet acc;

  for (int j = 0; j < n; ++j) {
    // ---- pivot search: izamax over rows j..n-1 of column j
    double bv = -1.0;
    int bi = n;
    for (int i = j + tid; i < n; i += blockDim.x) {
      double2 v = LU_A(i, j);
      double m = fabs(v.x) + fabs(v.y);
      if (m > bv) { bv = m; bi = i; }
    }
    for (int off = 16; off; off >>= 1) {
      double ov = __shfl_down_sync(0xffffffffu, bv, off);
      int oi = __shfl_down_sync(0xffffffffu, bi, off);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < nwarps ? red_v[lane] : -1.0;
      bi = lane < nwarps ? red_i[lane] : n;
      for (int off = 16; off; off >>= 1) {
        double ov = __shfl_down_sync(0xffffffffu, bv, off);
        int oi = __shfl_down_sync(0xffffffffu, bi, off);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0) s_piv = (bi < n) ? bi : j;   // NaN column: keep the diagonal
    }
    __syncthreads();
    const int piv = s_piv;
    // ---- row interchange (columns j..n-1; L columns are not needed for det)
    if (piv != j) {
      for (int c = j + tid; c < n; c += blockDim.x) {
        KLS_UNLESS(LU_IN(j, c) && LU_IN(piv, c), continue)
        double2 t = A[(size_t)j * n + c];
        A[(size_t)j * n + c] = A[(size_t)piv * n + c];
        A[(size_t)piv * n + c] = t;
      }
    }
    __syncthreads();
    // ---- pivot row and scaled column to shared memory
    double2 u = LU_A(j, j);
    const bool nz = (u.x != 0.0 || u.y != 0.0);
    double2 ru = nz ? cinv(u.x, u.y) : make_double2(0.0, 0.0);
    for (int c = j + 1 + tid; c < n; c += blockDim.x) prow[c] = LU_A(j, c);
    for (int i = j + 1 + tid; i < n; i += blockDim.x) lcol[i] = cmul(LU_A(i, j), ru);
    if (tid == 0) s_u = u;
    __syncthreads();
    // ---- rank-1 update of the trailing matrix
    for (int i = j + 1 + warp; i < n; i += nwarps) {
      double2 l = lcol[i];
      double2* row = A + (size_t)i * n;
      for (int c = j + 1 + lane; c < n; c += 32) {
        KLS_UNLESS(LU_IN(i, c), continue)
        double2 p = prow[c];
        double2 a = row[c];
        row[c] = lu_update(a, l, p);
      }
    }
    // ---- determinant accumulation (thread 0)
    if (tid == 0) acc.times(s_u, piv != j);
    __syncthreads();
  }
  if (tid == 0) acc.store(det_out, logabs_out);
}

__global__ void __launch_bounds__(LU_THREADS)
lu_det_kernel(int n, double2* __restrict__ Aall, double2* __restrict__ det_out,
              double* __restrict__ logabs_out) {
  extern __shared__ double2 sh[];        // prow[n], lcol[n]
  lu_det_body(n, Aall + (size_t)blockIdx.x * n * n, sh, det_out + blockIdx.x,
              logabs_out ? logabs_out + blockIdx.x : nullptr);
}

// one (model, omega) pair per CTA, matrices of different sizes
__global__ void __launch_bounds__(LU_THREADS)
multi_lu_kernel(const kls_mdesc* __restrict__ md, const int2* __restrict__ pairs) {
  extern __shared__ double2 sh[];
  const int2 pz = pairs[blockIdx.x];
  const kls_mdesc& d = md[pz.x];
  lu_det_body(d.Na, d.A + (size_t)pz.y * d.Na * d.Na, sh, d.det + pz.y, d.logabs + pz.y);
}

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
// Measured (1 matrix, B200): N = 101 312 -> 99 us, 201 557 -> 266 us, 301 1022 ->
// 558 us against one CTA (101) or a cluster with one barrier per column; 16
// matrices 315 -> 100, 612 -> 350, 2760 -> 1111 us.  A column's chain is about
// 1600 cycles at 4 rows a lane and 3300 at 10 (hand-over 160 / 360, update 280 / 540,
// pivot search with its reciprocal 670 / 1260, broadcast 60 / 80, multipliers and
// publication 440 / 1100; the marks themselves are some 50 each): about 350
// instructions that depend on one another.
constexpr int LUP_THREADS = 32 * LUP_WARPS;

struct LupMeta {
  double2 u;                  // pivot
  int piv, pos;               // its row, and that row's position before the exchange
};

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

__host__ __device__ inline size_t lup_smem(int n, int slots) {
  return (size_t)slots * ((size_t)n * sizeof(double2) + sizeof(LupMeta) + sizeof(uint64_t)) + 16;
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

// The size classes: rows per lane x columns per warp, CTAs per cluster.  4 columns
// a warp keep enough matrices on the device at once; a wider form (2 columns) for
// batches that it holds in one wave (7 matrices).  From <10,4> on, and a little in
// others, the registers do not hold all of it (142 bytes spilled a thread, <13,4> 1.0
// KB, <16,4> 2.2 KB).  1 matrix / 16, us:
//   N =  64  <2,2> x 4   53 /  53   (<2,8> x 1    71 /  71)
//   N = 101  <4,3> x 6   99 / 100   (<4,4> x 4   105 / 105, <4,2> x 8 128 / 249)
//   N = 192  <6,4> x 6  276 / 276   (<6,3> x 8   306 / 605), <6,2> x 12 236 / 693
//   N = 201  <7,5> x 6  350 / 350   (<7,4> x 8   333 / 656), <7,2> x 14 266 / 790
//   N = 256  <8,4> x 8  455 / 899   (<8,5> x 7   574 / 1140), <8,2> x 16 398 / 1181
//   N = 301 <10,4> x 10 558 / 1111  (<10,3> x 16 632 / 1887)
//   N = 400 <13,4> x 13 1250 / 3748 (<16,4> x 16 3277 / 9852)
//   N = 512 <16,4> x 16 2936 / 8782
// (in brackets: before the warp whose column is next polled)
struct LupClass {
  int n_max, C;
  const void *one, *multi;
  double us;                  // a wave of matrices, per column (lup_wins)
  int Cw;
  const void* wide;
};
#define LUP_CLASS(n, c, rpl, lp)                                                     \
  n, c, (const void*)lu_pipe_kernel<rpl, lp>, (const void*)multi_lu_pipe_kernel<rpl, lp>
const LupClass lup_classes[] = {
    {LUP_CLASS(64, 4, 2, 2), 0.84, 0, nullptr},
    {LUP_CLASS(128, 6, 4, 3), 1.08, 0, nullptr},
    {LUP_CLASS(192, 6, 6, 4), 1.41, 12, (const void*)lu_pipe_kernel<6, 2>},
    {LUP_CLASS(224, 6, 7, 5), 1.71, 14, (const void*)lu_pipe_kernel<7, 2>},
    {LUP_CLASS(256, 8, 8, 4), 1.77, 16, (const void*)lu_pipe_kernel<8, 2>},
    {LUP_CLASS(320, 10, 10, 4), 1.80, 0, nullptr},
    {LUP_CLASS(416, 13, 13, 4), 2.90, 0, nullptr},
    {LUP_CLASS(512, 16, 16, 4), 4.00, 0, nullptr},
};
#undef LUP_CLASS
constexpr int LUP_CLASSES = (int)(sizeof(lup_classes) / sizeof(lup_classes[0]));

// Ring slots: one per column where 200 KB hold them (N <= 112: no slot is
// written twice), else an even number of them, at least 16.
// Where a batch is more than one wave, half as many: the classes up to N = 128 then
// have two CTAs on an SM (63 matrices of N = 101: 290 -> 246 us).
int lup_slots(int n, bool half = false) {
  const int s = (int)((half ? 102400 : 204800) / (n * sizeof(double2) + 32));
  return n <= s ? n : std::max(16, s & ~1);
}

cudaLaunchConfig_t lup_config(int C, int matrices, size_t smem, cudaStream_t st,
                              cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.gridDim = dim3(C * matrices);
  cfg.blockDim = dim3(LUP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// shared-memory and cluster-size limits of a kernel (properties shared by every
// context in the process: always the largest value of the class)
cudaError_t lup_limits(const void* fn, int C) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024);
  if (e == cudaSuccess && C > 8)
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

}  // namespace

// clusters of C CTAs of fn that the device holds at once (0: none), with the whole ring
// or half of it
static int lup_clusters(const void* fn, int C, int n, bool half) {
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = lup_config(C, 1, lup_smem(n, lup_slots(n, half)), nullptr, &at);
  int clusters = 0;
  if (lup_limits(fn, C) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess)
    return clusters;
  cudaGetLastError();
  return 0;
}

// Size class of an n x n factorisation, -1 where there is none
static int lup_class(int n) {
  for (int k = 0; k < LUP_CLASSES; ++k)
    if (n <= lup_classes[k].n_max) return k;
  return -1;
}

static int lup_sms(int device) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

int kls_run_lu(kls_ctx* c, int n) {
  if (c->lu_mode != KLS_LU_CTA) {
    if (c->lu_class == -2) {
      c->lu_class = lup_class(c->Na);
      if (c->lu_class >= 0) {
        const LupClass& k = lup_classes[c->lu_class];
        c->lu_full = lup_clusters(k.one, k.C, c->Na, false);
        c->lu_half = lup_clusters(k.one, k.C, c->Na, true);
        c->lu_wide = k.wide ? lup_clusters(k.wide, k.Cw, c->Na, false) : 0;
        if (!c->lu_full) c->lu_class = -1;
      }
    }
    if (c->lu_class >= 0 &&
        (c->lu_mode == KLS_LU_CLUSTER ||
         lup_wins(n, c->Na, n <= c->lu_full ? c->lu_full : c->lu_half,
                  lup_classes[c->lu_class].us, lup_sms(c->device)))) {
      const LupClass& k = lup_classes[c->lu_class];
      const bool wide = n <= c->lu_wide;
      const int C = wide ? k.Cw : k.C;
      const int slots = lup_slots(c->Na, n > c->lu_full);
      cudaLaunchAttribute at;
      cudaLaunchConfig_t cfg = lup_config(C, n, lup_smem(c->Na, slots), c->stream, &at);
      const double2* A = c->d_A;
      KlsLuWait wait{c->lu_wait_ns, c->lu_skip};
      c->lu_skip = -1;
      void* args[] = {&c->Na, (void*)&slots, (void*)&C, &A, &c->d_det, &c->d_logabs, &wait};
      KLS_CK(c, cudaLaunchKernelExC(&cfg, wide ? k.wide : k.one, args));
      KLS_LAUNCHED(c);
      return KLS_OK;
    }
    if (c->lu_class < 0 && c->lu_mode == KLS_LU_CLUSTER)
      return kls_fail(c, KLS_ERR_UNSUPPORTED, "cluster LU does not fit this N_alpha");
  }
  size_t sm = 2 * (size_t)c->Na * sizeof(double2);
  if (sm > 48 * 1024)
    KLS_CK(c, cudaFuncSetAttribute(lu_det_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sm));
  lu_det_kernel<<<n, LU_THREADS, sm, c->stream>>>(c->Na, c->d_A, c->d_det, c->d_logabs);
  KLS_LAUNCHED(c);
  return KLS_OK;
}

// size class of a model's matrices for kls_multi_launch_lu (-1: one CTA each), on the
// current device
int kls_lu_class(int n) {
  const int k = lup_class(n);
  return k >= 0 && lup_clusters(lup_classes[k].multi, lup_classes[k].C, n, false) ? k : -1;
}
int kls_lu_classes() { return LUP_CLASSES; }

// the pairs of one size class (class -1, or where it is the slower one: lu_det_body,
// max_Na rows)
int kls_multi_launch_lu(cudaStream_t st, const kls_mdesc* d_md, const int2* d_pairs, int n_pairs,
                        int max_Na, int cls, const KlsLuWait& wait) {
  cudaError_t e;
  int device = 0;
  if ((e = cudaGetDevice(&device)) != cudaSuccess) return (int)e;
  // (its limits are those that kls_lu_class set)
  const int full = cls >= 0 ? lup_clusters(lup_classes[cls].multi, lup_classes[cls].C, max_Na, false)
                            : 0;
  const bool half = n_pairs > full;
  const int clusters =
      full && half ? lup_clusters(lup_classes[cls].multi, lup_classes[cls].C, max_Na, true) : full;
  if (full && lup_wins(n_pairs, max_Na, clusters, lup_classes[cls].us, lup_sms(device))) {
    const LupClass& k = lup_classes[cls];
    // one ring size for the class: as many slots as its largest matrix gets
    int slots = lup_slots(max_Na, half);
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = lup_config(k.C, n_pairs, lup_smem(max_Na, slots), st, &at);
    void* args[] = {&d_md, &d_pairs, (void*)&k.C, &slots, (void*)&wait};
    return (int)cudaLaunchKernelExC(&cfg, k.multi, args);
  }
  size_t sm = 2 * (size_t)max_Na * sizeof(double2);
  if (sm > 48 * 1024 &&
      (e = cudaFuncSetAttribute(multi_lu_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sm)) != cudaSuccess)
    return (int)e;
  multi_lu_kernel<<<n_pairs, LU_THREADS, sm, st>>>(d_md, d_pairs);
  return (int)cudaGetLastError();
}
