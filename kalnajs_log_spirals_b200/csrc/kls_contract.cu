// MatrixBuilder on the device (FP64 form).
//
//   M(omega)[b, a] = G N(a) sum_k W[k, b] w_k(omega) conj(W[k, a]),
//   w_k = DJ_p F0l[p,l] / den,  den = omega - Omega_res[p,l],
//   den := 1e-12 + 1e-12 i  when |den| < 1e-12
//
// (MatrixBuilder.jl:27-69, NL_julia_direct.jl:299-310).  The reference loops
// the n_l harmonics with one ZGEMM each, after materialising
// weight .* conj(W) for every harmonic; here the whole K = NPh * n_l
// reduction is one split-K contraction of the real table on the FP64 tensor
// pipe (DMMA m8n8k4) and the resonant weight is applied to the A fragment
// while it is loaded from shared memory, so the weighted copy never exists.
//
//   weights_kernel : w_k(omega) for a batch of omegas (kls_basis.cu)
//   contract_kernel: one triangle of T = sum_k w_k V_k^T V_k, 64 x 64 parts,
//                    cp.async 4-stage pipeline over 16-row slabs of the
//                    table, partial parts per K split written to a workspace
//   reduce_kernel  : deterministic sum over splits, T -> M * G * N(a), I - M
#include "kls_internal.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

namespace {

// not volatile: the scheduler may interleave independent DMMAs
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// ---- contraction -----------------------------------------------------------
// The alpha grid is symmetric, W(-alpha) = conj W(alpha), so the table holds
// the real numbers V[k][2p] = Re W, V[k][2p + 1] = Im W at the np = ceil(Na / 2)
// alphas >= 0 (kls_internal.cuh), and
//   T(omega) = sum_k w_k V[k]^T V[k],   complex symmetric, ldv x ldv,
// gives every entry of M: with W_b = c_b + i s_b (s odd in alpha)
//   sum_k w W_b conj(W_a) = T_cc + T_ss + i (T_sc - T_cs).
// Half the columns, real operands (one real product per component of w) and
// one triangle: 2 Na (Na + 1) flops per row of the table against the 8 Na^2 of
// the complex product.
//
// Bound: the FP64 tensor pipe (DMMA m8n8k4; 36.6 TFLOP/s measured with all
// warps issuing).  T is cut into 8 x 8 blocks; 8 blocks make a group, and a
// CTA of 4 warps takes the part (gi, gj <= gi) of the triangle for one range
// of k: 64 x 64 off the diagonal (a warp: 4 x 4 blocks), the 36 lower blocks on
// it (a warp: block rows w and 7 - w, 9 blocks each).  Only the last group may
// be narrower, so its work is its blocks' work to within one block row: 741
// blocks at Na = 301 cost 187 x 4 (a 64 x 64 tiling of the triangle: 240 x 4).
constexpr int CT_BK = 16;                   // table rows per slab
constexpr int CT_S = 68;                    // doubles per slab row: conflict-free fragments
constexpr int CT_STAGES = 4;
constexpr int CT_THREADS = 128;
constexpr int CT_PLANE = CT_BK * CT_S;      // doubles per side per stage
constexpr int CT_STAGE_DOUBLES = 2 * CT_PLANE + 2 * CT_BK;
constexpr size_t CT_SMEM = (size_t)CT_STAGES * CT_STAGE_DOUBLES * sizeof(double);
constexpr int CT_SLOT = 64 * 64;            // complex values of one partial tile

struct CtItem {
  int gi, gj;                // groups of the block rows and columns
  int n8;                    // 8-blocks of T in all
  int64_t k0;                // first table row
  int nk;                    // slabs
  int64_t K_pad;
  int ldv;
};

// The slab pipeline shared by every tile shape: the callers differ per warp in
// what `mma` does with a slab, and the barrier counts warps, not places.
template <typename F>
__device__ __forceinline__ void ct_pipeline(const CtItem& it, const double* __restrict__ V,
                                            const double2* __restrict__ wz, double* smem, F mma) {
  const int tid = threadIdx.x;
  const int rows8 = min(8, it.n8 - 8 * it.gi);         // blocks of the row group
  const bool diag = it.gi == it.gj;
  const int c0r = it.gi * 64, c0c = it.gj * 64;
  const int row_chunks = rows8 * 4;                    // 16-byte chunks per row
  auto load = [&](int s, int kt) {
    double* st = smem + (size_t)s * CT_STAGE_DOUBLES;
    const int64_t k0 = it.k0 + (int64_t)kt * CT_BK;
    const double* src = V + (size_t)k0 * it.ldv;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = tid + q * CT_THREADS;              // 0..511
      const int r = e >> 5, c = e & 31;
      if (c < row_chunks)
        KLS_IF(KLS_IB((k0 + r) * (int64_t)it.ldv + c0r + 2 * c + 1, it.K_pad * it.ldv,
                      KS_CONTRACT_SRC))
        cp_async16(st + r * CT_S + 2 * c, src + (size_t)r * it.ldv + c0r + 2 * c);
      if (!diag)
        KLS_IF(KLS_IB((k0 + r) * (int64_t)it.ldv + c0c + 2 * c + 1, it.K_pad * it.ldv,
                      KS_CONTRACT_SRC))
        cp_async16(st + CT_PLANE + r * CT_S + 2 * c, src + (size_t)r * it.ldv + c0c + 2 * c);
    }
    if (tid < CT_BK) KLS_IF(KLS_IB(k0 + tid, it.K_pad, KS_CONTRACT_SRC))
      cp_async16(st + 2 * CT_PLANE + 2 * tid, wz + k0 + tid);
  };
#pragma unroll
  for (int s = 0; s < CT_STAGES - 1; ++s) {
    if (s < it.nk) load(s, s);
    cp_async_commit();
  }
  for (int kt = 0; kt < it.nk; ++kt) {
    cp_async_wait<CT_STAGES - 2>();
    asm volatile("bar.sync 0, %0;" ::"n"(CT_THREADS) : "memory");
    const int nxt = kt + CT_STAGES - 1;
    if (nxt < it.nk) load(nxt % CT_STAGES, nxt);
    cp_async_commit();
    mma(smem + (size_t)(kt % CT_STAGES) * CT_STAGE_DOUBLES);
  }
  cp_async_wait<0>();
}

// one 8 x 8 block of a partial tile: 64 complex values in row order
__device__ __forceinline__ void ct_store(double2* __restrict__ out, int bi, int bj, double r0,
                                         double r1, double i0, double i1) {
  const int lane = threadIdx.x & 31;
  double2* o = out + (bi * 8 + bj) * 64 + 2 * lane;
  o[0] = make_double2(r0, i0);
  o[1] = make_double2(r1, i1);
}

// NR x 4 blocks of an off-diagonal part, from block row r0 and block column c0
template <int NR>
__device__ __forceinline__ void ct_off(const CtItem& it, const double* __restrict__ V,
                                       const double2* __restrict__ wz, double2* __restrict__ out,
                                       double* smem, int r0, int c0) {
  constexpr int N1 = NR > 0 ? NR : 1;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double cr[N1][4][2], ci[N1][4][2];
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;
  ct_pipeline(it, V, wz, smem, [&](const double* st) {
    if (NR == 0) return;
    const double* sA = st + r0 * 8 + g;
    const double* sB = st + CT_PLANE + c0 * 8 + g;
    const double* sd = st + 2 * CT_PLANE;
#pragma unroll
    for (int kk = 0; kk < CT_BK; kk += 4) {
      const int kr = kk + t;
      const double dr = sd[2 * kr], di = sd[2 * kr + 1];
      double ar[N1], ai[N1], b[4];
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const double x = sA[kr * CT_S + i * 8];
        ar[i] = dr * x;
        ai[i] = di * x;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = sB[kr * CT_S + j * 8];
#pragma unroll
      for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dmma(cr[i][j][0], cr[i][j][1], ar[i], b[j]);
          dmma(ci[i][j][0], ci[i][j][1], ai[i], b[j]);
        }
    }
  });
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      ct_store(out, r0 + i, c0 + j, cr[i][j][0], cr[i][j][1], ci[i][j][0], ci[i][j][1]);
}

// The lower blocks of a diagonal part of N block rows: warp W takes block rows
// N - 1 - W (blocks 0 .. N - 1 - W) and W (blocks 0 .. W), N + 1 blocks in all;
// an odd N leaves its middle row to one warp.  A block row's A fragment is the
// same block column's B fragment, so a slab row is read once.
template <int N, int W>
__device__ __forceinline__ void ct_diag(const CtItem& it, const double* __restrict__ V,
                                        const double2* __restrict__ wz, double2* __restrict__ out,
                                        double* smem) {
  constexpr int HI = N - 1 - W, LO = W;
  constexpr int NH = HI >= LO ? HI + 1 : 0, NL = HI > LO ? LO + 1 : 0, NS = NH + NL;
  constexpr int N1 = NS > 0 ? NS : 1, H = HI > 0 ? HI : 0, L = NL ? LO : 0;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double cr[N1][2], ci[N1][2];
#pragma unroll
  for (int s = 0; s < NS; ++s) cr[s][0] = cr[s][1] = ci[s][0] = ci[s][1] = 0.0;
  ct_pipeline(it, V, wz, smem, [&](const double* st) {
    if (NS == 0) return;
    const double* sv = st + g;
    const double* sd = st + 2 * CT_PLANE;
#pragma unroll
    for (int kk = 0; kk < CT_BK; kk += 4) {
      const int kr = kk + t;
      const double dr = sd[2 * kr], di = sd[2 * kr + 1];
      double b[H + 1];
#pragma unroll
      for (int j = 0; j <= H; ++j) b[j] = sv[kr * CT_S + j * 8];
      const double hr = dr * b[H], hi = di * b[H], lr = dr * b[L], li = di * b[L];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double x = b[s < NH ? s : s - NH];
        dmma(cr[s][0], cr[s][1], s < NH ? hr : lr, x);
        dmma(ci[s][0], ci[s][1], s < NH ? hi : li, x);
      }
    }
  });
#pragma unroll
  for (int s = 0; s < NS; ++s)
    ct_store(out, s < NH ? H : L, s < NH ? s : s - NH, cr[s][0], cr[s][1], ci[s][0], ci[s][1]);
}

template <int N>
__device__ __forceinline__ void ct_diag_warp(const CtItem& it, const double* __restrict__ V,
                                             const double2* __restrict__ wz,
                                             double2* __restrict__ out, double* smem) {
  switch (threadIdx.x >> 5) {
    case 0: ct_diag<N, 0>(it, V, wz, out, smem); break;
    case 1: ct_diag<N, 1>(it, V, wz, out, smem); break;
    case 2: ct_diag<N, 2>(it, V, wz, out, smem); break;
    default: ct_diag<N, 3>(it, V, wz, out, smem); break;
  }
}

// one partial tile: out = this item's 64 x 64 slot (64-value blocks in row order)
__device__ __forceinline__ void ct_item(const CtItem& it, const double* __restrict__ V,
                                        const double2* __restrict__ wz, double2* __restrict__ out,
                                        double* smem) {
  const int warp = threadIdx.x >> 5;
  const int n = min(8, it.n8 - 8 * it.gi);
  if (it.gi == it.gj) {
    switch (n) {
      case 8: ct_diag_warp<8>(it, V, wz, out, smem); break;
      case 7: ct_diag_warp<7>(it, V, wz, out, smem); break;
      case 6: ct_diag_warp<6>(it, V, wz, out, smem); break;
      case 5: ct_diag_warp<5>(it, V, wz, out, smem); break;
      case 4: ct_diag_warp<4>(it, V, wz, out, smem); break;
      case 3: ct_diag_warp<3>(it, V, wz, out, smem); break;
      case 2: ct_diag_warp<2>(it, V, wz, out, smem); break;
      default: ct_diag_warp<1>(it, V, wz, out, smem); break;
    }
    return;
  }
  const int c0 = (warp & 1) * 4, half = (n + 1) >> 1;
  const int r0 = (warp >> 1) ? half : 0, nr = (warp >> 1) ? n - half : half;
  switch (nr) {
    case 4: ct_off<4>(it, V, wz, out, smem, r0, c0); break;
    case 3: ct_off<3>(it, V, wz, out, smem, r0, c0); break;
    case 2: ct_off<2>(it, V, wz, out, smem, r0, c0); break;
    case 1: ct_off<1>(it, V, wz, out, smem, r0, c0); break;
    default: ct_off<0>(it, V, wz, out, smem, r0, c0); break;
  }
}

// items: (gi << 16 | gj, slot, first slab, slabs)
__global__ void __launch_bounds__(CT_THREADS, 2)
contract_kernel(int n8, int ldv, int64_t K_pad, int n_slots, const int4* __restrict__ items,
                const double* __restrict__ V, const double2* __restrict__ wt,
                double2* __restrict__ part) {
  extern __shared__ __align__(16) double smem[];
  const int4 q = items[blockIdx.x];
  KLS_UNLESS(KLS_IB(q.y, n_slots, KS_CONTRACT_OUT), return)
  CtItem it{q.x >> 16, q.x & 0xffff, n8, (int64_t)q.z * CT_BK, q.w, K_pad, ldv};
  ct_item(it, V, wt + (size_t)blockIdx.y * K_pad,
          part + ((size_t)blockIdx.y * n_slots + q.y) * CT_SLOT, smem);
}

// Persistent form over an uneven batch: every CTA takes work items
// (model, omega, part, range of k) from an atomic counter until the list is
// exhausted.  The list runs model by model, largest first, so CTAs running
// together share a k-range of one table (L2 reuse) and the tail of the launch
// is made of the small models' items.  Each item computes exactly what
// contract_kernel computes for it, so a determinant is bitwise the same.
__global__ void __launch_bounds__(CT_THREADS, 2)
multi_contract_kernel(const kls_mdesc* __restrict__ md, const kls_item* __restrict__ items,
                      int n_items, int* __restrict__ counter) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int i = s_item;
    if (i >= n_items) break;
    const kls_item q = items[i];
    const kls_mdesc& d = md[q.model];
    KLS_IF(KLS_IB(q.split, d.n_slots, KS_CONTRACT_OUT)) {
      CtItem it{q.tile >> 16, q.tile & 0xffff, d.ldv / 8, (int64_t)q.kb0 * CT_BK, q.nkb, d.K_pad,
                d.ldv};
      ct_item(it, d.V, d.wt + (size_t)q.z * d.K_pad,
              d.part + ((size_t)q.z * d.n_slots + q.split) * CT_SLOT, smem);
    }
    __syncthreads();          // shared stages and s_item are reused by the next item
  }
}

// ---- split reduction + epilogue ------------------------------------------------
// One CTA per 8 x 8 block of T (4 x 4 pairs of alphas): 16 threads per pair sum
// its 2 x 2 values over every 16th partial, the 16 sums are added in order, and
// the pair's up to 8 entries of M (signs of the two alphas, both triangles)
// come out of them.  Bound by the partials' bytes, read once.
constexpr int RD_THREADS = 256;

__device__ __forceinline__ int alpha_index(int N, int p, bool pos) {
  const int np = (N + 1) >> 1;
  if (N & 1) return pos ? np - 1 + p : np - 1 - p;
  return pos ? np + p : np - 1 - p;
}

__device__ __forceinline__ void reduce_body(int Na, int blk, double G,
                                            const double* __restrict__ Nk,
                                            const int2* __restrict__ tiles, int n_slots,
                                            const double2* __restrict__ part,
                                            double2* __restrict__ A, double2* __restrict__ Mout) {
  __shared__ double sm[16][16][9];
  __shared__ double tot[16][8];
  // block (bi, bj <= bi) of the triangle
  int bi = (int)((sqrtf(8.f * (float)blk + 1.f) - 1.f) * 0.5f);
  while ((bi + 1) * (bi + 2) / 2 <= blk) ++bi;
  while (bi * (bi + 1) / 2 > blk) --bi;
  const int bj = blk - bi * (bi + 1) / 2;
  const int gi = bi >> 3, gj = bj >> 3;
  const int2 tl = tiles[gi * (gi + 1) / 2 + gj];       // (first slot, slots)
  const int tid = threadIdx.x, pr = tid & 15, sg = tid >> 4;
  const int pi = pr >> 2, qi = pr & 3;
  const double2* src = part + (size_t)tl.x * CT_SLOT + ((bi & 7) * 8 + (bj & 7)) * 64 + pi * 16 +
                       qi * 2;
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 2
  for (int s = sg; s < tl.y; s += 16) {
    KLS_UNLESS(KLS_IB(tl.x + s, n_slots, KS_REDUCE), continue)
    const double2* p = src + (size_t)s * CT_SLOT;
    const double2 a = p[0], b = p[1], c = p[8], d = p[9];
    v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
    v[4] += c.x; v[5] += c.y; v[6] += d.x; v[7] += d.y;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) sm[sg][pr][e] = v[e];
  __syncthreads();
  if (tid >= 128) {
    const int q = (tid - 128) >> 3, e = tid & 7;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += sm[k][q][e];
    tot[q][e] = s;
  }
  __syncthreads();
  if (tid >= 128) return;
  const int q16 = tid >> 3, o = tid & 7;
  const int p = 4 * bi + (q16 >> 2), q = 4 * bj + (q16 & 3);
  const int np = (Na + 1) >> 1;
  const bool swap = o & 4, sb = !(o & 2), sa = !(o & 1);   // alpha_b, alpha_a >= 0
  if (p < q || p >= np || (swap && p == q)) return;
  const int P = swap ? q : p, Q = swap ? p : q;
  if ((Na & 1) && ((P == 0 && !sb) || (Q == 0 && !sa))) return;
  const double* T = tot[q16];
  const double ccr = T[0], cci = T[1], ssr = T[6], ssi = T[7];
  const double scr = swap ? T[2] : T[4], sci = swap ? T[3] : T[5];   // Im W_b Re W_a
  const double csr = swap ? T[4] : T[2], csi = swap ? T[5] : T[3];   // Re W_b Im W_a
  const double fb = sb ? 1.0 : -1.0, fa = sa ? 1.0 : -1.0, f = sb == sa ? 1.0 : -1.0;
  const double sr = (ccr + f * ssr) - (fb * sci - fa * csi);
  const double si = (cci + f * ssi) + (fb * scr - fa * csr);
  const int b = alpha_index(Na, P, sb), a = alpha_index(Na, Q, sa);
  const double n = Nk[a];
  // unfused products: 1 - mr must not become an FMA in one kernel only
  const double mr = __dmul_rn(__dmul_rn(sr, G), n), mi = __dmul_rn(__dmul_rn(si, G), n);
  const size_t e = (size_t)b * Na + a;
  KLS_UNLESS(KLS_IB(e, (int64_t)Na * Na, KS_REDUCE), return)
  A[e] = make_double2((a == b ? 1.0 : 0.0) - mr, -mi);
  if (Mout) Mout[e] = make_double2(mr, mi);
}

__global__ void __launch_bounds__(RD_THREADS)
reduce_kernel(int Na, double G, const double* __restrict__ Nk, const int2* __restrict__ tiles,
              int n_slots, const double2* __restrict__ part, double2* __restrict__ A,
              double2* __restrict__ Mout) {
  const int z = blockIdx.y;
  reduce_body(Na, blockIdx.x, G, Nk, tiles, n_slots, part + (size_t)z * n_slots * CT_SLOT,
              A + (size_t)z * Na * Na, z == 0 ? Mout : nullptr);
}

__global__ void __launch_bounds__(RD_THREADS)
multi_reduce_kernel(const kls_mdesc* __restrict__ md, const int2* __restrict__ pairs) {
  const int2 pz = pairs[blockIdx.y];
  const kls_mdesc& d = md[pz.x];
  const int n8 = d.ldv / 8;
  if ((int)blockIdx.x >= n8 * (n8 + 1) / 2) return;
  reduce_body(d.Na, blockIdx.x, d.G, d.Nk, d.tiles, d.n_slots,
              d.part + (size_t)pz.y * d.n_slots * CT_SLOT, d.A + (size_t)pz.y * d.Na * d.Na,
              nullptr);
}

}  // namespace

// CTAs of the FP64 contraction resident on the device at once
static int f64_slots(int device, bool persistent) {
  int sms = 148, per_sm = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const void* fn = persistent ? (const void*)multi_contract_kernel : (const void*)contract_kernel;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CT_SMEM);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, CT_THREADS, CT_SMEM) !=
          cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  return sms * per_sm;
}

// Time per slab of part (gi, gj), full off-diagonal part = 160: the blocks of
// the busiest warp, and 8% more per block on the diagonal (two weighted rows
// for 9 blocks; 30.5 TFLOP/s against 32.9 off it, 6 us to 1 ms items).
static int part_cost(int n8, int gi, int gj) {
  const int n = std::min(8, n8 - 8 * gi);
  return gi == gj ? 54 * (n > 1 ? n + 1 : 1) / 5 : 40 * ((n + 1) / 2);
}

// K splits of a part when a full off-diagonal one takes `splits`: in proportion
// to its cost, so that the items of the launch take the same time.
static int part_splits(int cost, int splits, int64_t slabs) {
  const int64_t s = ((int64_t)splits * cost + 80) / 160;
  return (int)std::max<int64_t>(1, std::min<int64_t>(s, slabs));
}

// Of n >= 6 splits the last 2/5 are a third as long as the others and run
// last, so the launch's tail is a third of an item: first slab of split j.
static int64_t split_begin(int64_t slabs, int n, int j) {
  const int big = n >= 6 ? 3 * n / 5 : n;
  const int64_t units = 3 * (int64_t)big + (n - big);
  const int64_t at = j <= big ? 3 * (int64_t)j : 3 * (int64_t)big + (j - big);
  return slabs * at / units;
}

// a split has at least 4 slabs
int kls_f64_max_splits(const kls_ctx* c) {
  if (c->sim) return kls_similar_max_splits(c);
  return (int)std::max<int64_t>(1, std::min<int64_t>(c->K_pad / (4 * CT_BK), INT_MAX / 1024));
}

// The split count depends on the table and the device only, never on the
// batch size, so a determinant is bitwise identical whichever batch it is
// evaluated in.  It minimises the estimated time of one omega: the items' work
// over the resident CTAs, an item's fixed cost (pipeline fill, its 64 KB
// partial written and read back: about 4 slabs' time) and 0.4 of a last item
// in the tail (measured: 214,272 rows at Na = 301 took 1.635 / 1.463 / 1.341 ms
// with 470 / 935 / 2071 equal items, 1.28 without a tail).  At most 4096 items
// (268 MB of partials per omega).
int kls_choose_splits(const kls_ctx* c) {
  if (c->sim) return kls_similar_splits(c);
  const int n8 = c->ldv / 8, G = (n8 + 7) / 8;
  const int slots = f64_slots(c->device, false);
  const int64_t slabs = c->K_pad / CT_BK;
  const int max_s = std::min(kls_f64_max_splits(c), 4096);
  const double fixed = 4 * 160.0;
  int best = 1;
  double best_t = INFINITY;
  for (int s = 1; s <= max_s; ++s) {
    int64_t items = 0;
    double work = 0.0, first = 0.0, last = 0.0;
    // the last group's parts differ from the others; each kind once
    auto add = [&](int64_t count, int gi, int gj) {
      if (count <= 0) return;
      const int cost = part_cost(n8, gi, gj), n = part_splits(cost, s, slabs);
      items += count * n;
      work += (double)count * cost * slabs;
      first = std::max(first, (double)cost * (double)split_begin(slabs, n, 1));
      last = std::max(last, (double)cost * (double)(slabs - split_begin(slabs, n, n - 1)));
    };
    const int64_t full = G - 1;
    add(full * (full - 1) / 2, 1, 0);
    add(full, 0, 0);
    add(full, G - 1, 0);
    add(1, G - 1, G - 1);
    if (s > 1 && items > 4096) break;
    const double spread = (work + items * fixed) / slots;
    const double t = items <= slots ? 1.1 * first + fixed : std::max(spread, first) + 0.4 * last + fixed;
    if (t < best_t) { best_t = t; best = s; }
  }
  return best;
}

// Items and slots of the context's split count, on the host and the device.
// Long items come first, each kind ordered by where in k it starts, so CTAs
// running together read the same rows of the table.
int kls_f64_plan(kls_ctx* c) {
  if (c->plan_splits == c->splits) return KLS_OK;
  const int n8 = c->ldv / 8, G = (n8 + 7) / 8;
  const int64_t slabs = c->K_pad / CT_BK;
  std::vector<int4> items, tail;
  std::vector<int2> tiles;
  int slot = 0;
  for (int gi = 0; gi < G; ++gi)
    for (int gj = 0; gj <= gi; ++gj) {
      const int n = part_splits(part_cost(n8, gi, gj), c->splits, slabs);
      tiles.push_back(make_int2(slot, n));
      for (int s = 0; s < n; ++s) {
        const int64_t b = split_begin(slabs, n, s), e = split_begin(slabs, n, s + 1);
        (n >= 6 && s >= 3 * n / 5 ? tail : items)
            .push_back(make_int4(gi << 16 | gj, slot++, (int)b, (int)(e - b)));
      }
    }
  auto by_k = [](const int4& a, const int4& b) { return a.z < b.z; };
  std::stable_sort(items.begin(), items.end(), by_k);
  std::stable_sort(tail.begin(), tail.end(), by_k);
  items.insert(items.end(), tail.begin(), tail.end());
  cudaFree(c->d_items);
  cudaFree(c->d_tiles);
  c->d_items = nullptr;
  c->d_tiles = nullptr;
  c->plan_splits = 0;
  KLS_CK(c, cudaMalloc(&c->d_items, items.size() * sizeof(int4)));
  KLS_CK(c, cudaMalloc(&c->d_tiles, tiles.size() * sizeof(int2)));
  KLS_CK(c, cudaMemcpyAsync(c->d_items, items.data(), items.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, c->stream));
  KLS_CK(c, cudaMemcpyAsync(c->d_tiles, tiles.data(), tiles.size() * sizeof(int2),
                            cudaMemcpyHostToDevice, c->stream));
  KLS_CK(c, cudaStreamSynchronize(c->stream));   // an uneven batch copies them on its own stream
  c->items.swap(items);
  c->n_slots = slot;
  c->plan_splits = c->splits;
  return KLS_OK;
}

size_t kls_f64_part_elems(const kls_ctx* c, int n) { return (size_t)n * c->n_slots * CT_SLOT; }

int kls_run_contract_f64(kls_ctx* c, int n) {
  KLS_CK(c, cudaFuncSetAttribute(contract_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)CT_SMEM));
  contract_kernel<<<dim3((unsigned)c->items.size(), n), CT_THREADS, CT_SMEM, c->stream>>>(
      c->ldv / 8, c->ldv, c->K_pad, c->n_slots, c->d_items, c->d_V, c->d_wt, c->d_part);
  KLS_LAUNCHED(c);
  return KLS_OK;
}

int kls_run_reduce(kls_ctx* c, int n, bool export_M) {
  const int n8 = c->ldv / 8;
  reduce_kernel<<<dim3(n8 * (n8 + 1) / 2, n), RD_THREADS, 0, c->stream>>>(
      c->Na, c->cfg.G, c->d_N, c->d_tiles, c->n_slots, c->d_part, c->d_A,
      export_M ? c->d_M : nullptr);
  KLS_LAUNCHED(c);
  return KLS_OK;
}

// ---- uneven batch over models (kls_multi.cu) ------------------------------------
int kls_multi_launch_f64(cudaStream_t st, const kls_mdesc* d_md, const int2* d_pairs, int n_pairs,
                         const kls_item* d_items, int n_items, int* d_counter, int grid,
                         int max_ldv) {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(multi_contract_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)CT_SMEM)) != cudaSuccess)
    return (int)e;
  if ((e = cudaMemsetAsync(d_counter, 0, sizeof(int), st)) != cudaSuccess) return (int)e;
  multi_contract_kernel<<<grid, CT_THREADS, CT_SMEM, st>>>(d_md, d_items, n_items, d_counter);
  if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  const int n8 = max_ldv / 8;
  multi_reduce_kernel<<<dim3(n8 * (n8 + 1) / 2, n_pairs), RD_THREADS, 0, st>>>(d_md, d_pairs);
  return (int)cudaGetLastError();
}

int kls_multi_contract_slots(int device) { return f64_slots(device, true); }
