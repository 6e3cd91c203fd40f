// M(omega) from the self-similarity of the orbits (FP64).
//
// The potential is ln r, so an orbit of eccentricity e at guiding radius Rc is
// the orbit at Rc = 1 scaled by Rc in r and in time.  With e and v the same for
// every Rc of the grid, the orbits of one column ie share w1, theta and r / Rc,
// and
//   W_l(alpha; Rc, e) = Rc^-1/2 e^{-i alpha ln Rc} What_l(alpha; e).
// With the uniform alpha grid (step da, indices b, a) the sum over the radii
// becomes one function of b - a per (l, e):
//   sum_k W[k,b] w_k conj W[k,a] = sum_{l,e} What_b conj(What_a) F_{l,e}(b - a),
//   F_{l,e}(d) = sum_R w(l, e, R) / Rc e^{-i d da ln Rc}.
// The frequencies, and with them the weights w, stay those of the single orbits.
//
// The computed orbits are similar to their rounding only: v_r^2 = 2 (E - ln r) -
// L^2 / r^2 cancels at the turning points, and the last bits of E and L^2 (two
// numbers per orbit) move w1 and theta by up to 1e-7.  So a column's samples are
// taken as x_R = x + u_R x_u + v_R x_v: mean, and the two directions of largest
// variance over the radii, with u, v per orbit.  To first order
//   What_R = What + u_R D_u + v_R D_v,
// which adds two channels (weights u w and v w) to F.  Every orbit of non-zero
// weight is compared with its column's form; where one does not fit (an orbit
// that a threshold of the integrator treats differently, for one), the model
// keeps the general table and contraction (kls_contract.cu).
//
//   fourier_kernel : F for the three channels, a GEMM of the weights
//                    [n_l Ne x NR] with the phases [NR x 2 N_alpha] (DMMA)
//   pair_kernel    : sum over (l, e) for the pairs of alphas
//   pair_reduce    : sum over the row splits, * G * N(a), I - M
//
// Work per omega: 12 n_l Ne NR N_alpha flops in F and 12 FP64 and 32 FP32 FMA per
// pair and (l, e) row over N_alpha^2 / 4 pairs, against 2 N_alpha^2 n_l Ne NR for the
// table: at NR = 501, Ne = 51, N_alpha = 301, l = +-100 1.9e10, 5.6e9 and 1.5e10
// against 9.3e11.
#include "kls_internal.cuh"
#include "kls_tcgen05.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

struct kls_similar {
  void* slab = nullptr;       // the arrays below, slab_bytes in all
  size_t slab_bytes = 0;
  int R = 0;                  // rows (l, e): il * Ne + ie
  int Nap = 0;                // N_alpha padded to the pair tiles
  int K2p = 0;                // mirrored pairs of radii, padded to the slabs of fourier_kernel
  double* V = nullptr;        // [R][ldv] What, pairs (Re, Im) at the alphas >= 0
  float2* Vf = nullptr;       // [R][ldv / 2] the same in FP32
  float4* D = nullptr;        // [R][ldv / 2] Re D_u, Re D_v, Im D_u, Im D_v
  double* U = nullptr;        // [3][Ne][NR] 1 / Rc, u / Rc, v / Rc
  double* Phi = nullptr;      // [2][K2p][Nap] cos, sin(d x da dln): x from the grid's centre
  double2* rot = nullptr;     // [Nap] cos, sin(d da ln Rc at the centre)
  int4* tiles = nullptr;      // pair tiles: I, J, weight (16: a full one), limit of q + p
  int n_tiles = 0;
  std::vector<int> weight;    // of the tiles
};

namespace {

// element i of an array of n, guarded in the bounds-checked build: arrays of the
// preparation, and of the evaluation
#define SIM_IN(i, n) KLS_IB((int64_t)(i), (int64_t)(n), KS_SIMILAR_PREP)
#define SIM_AT(i, n) KLS_IB((int64_t)(i), (int64_t)(n), KS_SIMILAR)

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}
// copies of 16 / 8 bytes; `n` = 0 writes zeros and reads nothing
__device__ __forceinline__ void cp16z(void* smem, const void* gmem, int n) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp8z(void* smem, const void* gmem, int n) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// ---- the columns' common orbits ----------------------------------------------
constexpr int SIM_PROBES = 6;     // w1 and theta at 3 samples: where u, v are read off
constexpr double SIM_H = 1e-5;    // step of the central differences behind D_u, D_v
// Accepted misfits of a column, relative to its max |What|: of its orbits'
// samples against their common form (on average and for any orbit), second
// order in (u, v), and the size of the first-order terms, which are summed in
// FP32.  Measured on the default grid: 2e-13 on average (2e-12 in the column
// nearest to circular), 1.3e-11 for the worst of 25,551 orbits, 1.5e-13 and
// 6e-8; an orbit of another branch misses by O(1).
constexpr double SIM_FIT = 1e-11, SIM_WORST = 1e-10, SIM_SECOND = 1e-12, SIM_FIRST = 1e-6;

__host__ __device__ inline int probe_at(int nwa, int q) {
  const int k = q == 0 ? nwa / 10 : q == 1 ? nwa / 2 : nwa - 1 - nwa / 10;
  return k < 1 ? (nwa > 1 ? 1 : 0) : (k > nwa - 2 && nwa > 2 ? nwa - 2 : k);
}

// per orbit: does it carry weight, and its probes and Omega_2 / Omega_1
__global__ void probe_kernel(int NPh, int nwa, const double* __restrict__ of,
                             const int* __restrict__ valid, const double* __restrict__ w1,
                             const double* __restrict__ pha, double* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NPh) return;
  KLS_UNLESS(SIM_IN((int64_t)OF_DJ * NPh + p, (int64_t)OF_COUNT * NPh), return)
  const double FE = of[(size_t)OF_FE * NPh + p], FL = of[(size_t)OF_FL * NPh + p];
  const double DJ = of[(size_t)OF_DJ * NPh + p];
  double* o = out + (size_t)p * (SIM_PROBES + 2);
  o[0] = valid[p] && !((FE == 0.0 && FL == 0.0) || DJ == 0.0) ? 1.0 : 0.0;
  o[1] = of[(size_t)OF_OM2 * NPh + p] / of[(size_t)OF_OM1 * NPh + p];
  for (int q = 0; q < 3; ++q) {
    const size_t k = (size_t)p * nwa + probe_at(nwa, q);
    KLS_UNLESS(SIM_IN(k, (int64_t)NPh * nwa), continue)
    o[2 + q] = w1[k];
    o[5 + q] = pha[k];
  }
}

// per (column, sample): mean and the slopes along u and v over the column's
// weighted orbits.  fit: [7][Ne][nwa] = w1, its slopes, theta, its slopes, r / Rc
__global__ void fit_kernel(int NR, int Ne, int nwa, const double* __restrict__ probes,
                           const double* __restrict__ U, const double2* __restrict__ inv_var,
                           const double* __restrict__ rc, const double* __restrict__ w1,
                           const double* __restrict__ ra, const double* __restrict__ pha,
                           double* __restrict__ fit) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x, ie = blockIdx.y;
  if (k >= nwa) return;
  double w0 = 0.0, p0 = 0.0, sw = 0.0, sp = 0.0, sr = 0.0, n = 0.0;
  double wu = 0.0, wv = 0.0, pu = 0.0, pv = 0.0;
  for (int iR = 0; iR < NR; ++iR) {
    const int p = iR + NR * ie;
    if (probes[(size_t)p * (SIM_PROBES + 2)] == 0.0) continue;
    const size_t e = (size_t)p * nwa + k;
    KLS_UNLESS(SIM_IN(e, (int64_t)NR * Ne * nwa), continue)
    const double w = w1[e], t = pha[e], u = U[p], v = U[(size_t)NR * Ne + p];
    if (n == 0.0) { w0 = w; p0 = t; }
    const double dw = w - w0, dp = t - p0;       // differences of near equals: exact
    sw += dw; sp += dp; sr += ra[e] / rc[iR]; n += 1.0;
    wu += dw * u; wv += dw * v; pu += dp * u; pv += dp * v;
  }
  const double2 iv = inv_var[ie];
  const size_t pl = (size_t)Ne * nwa, o = (size_t)ie * nwa + k;
  const double d = n > 0.0 ? 1.0 / n : 0.0;
  KLS_UNLESS(SIM_IN(6 * pl + o, 7 * pl), return)
  fit[o] = w0 + sw * d;
  fit[pl + o] = wu * iv.x;
  fit[2 * pl + o] = wv * iv.y;
  fit[3 * pl + o] = p0 + sp * d;
  fit[4 * pl + o] = pu * iv.x;
  fit[5 * pl + o] = pv * iv.y;
  fit[6 * pl + o] = n > 0.0 ? sr * d : 1.0;
}

// An orbit's misfit against its column's form, averaged over its samples: of w1
// (times l it is a phase), and of the rest of the integrand's phase and modulus
__global__ void misfit_kernel(int NR, int Ne, int nwa, double m, double amax,
                              const double* __restrict__ probes, const double* __restrict__ U,
                              const double* __restrict__ ratio_fit, const double* __restrict__ rc,
                              const double* __restrict__ w1, const double* __restrict__ ra,
                              const double* __restrict__ pha, const double* __restrict__ fit,
                              double2* __restrict__ out) {
  const int p = blockIdx.x, ie = p / NR, iR = p % NR;
  KLS_UNLESS(SIM_IN(p, NR * Ne), return)
  const double* pr = probes + (size_t)p * (SIM_PROBES + 2);
  if (pr[0] == 0.0) {
    if (threadIdx.x == 0) out[p] = make_double2(0.0, 0.0);
    return;
  }
  const double u = U[p], v = U[(size_t)NR * Ne + p];
  const double* rf = ratio_fit + 3 * ie;
  const double dq = fabs(pr[1] - (rf[0] + u * rf[1] + v * rf[2])), q = fabs(pr[1]);
  const size_t pl = (size_t)Ne * nwa;
  const double* f = fit + (size_t)ie * nwa;
  double a = 0.0, b = 0.0;
  for (int k = threadIdx.x; k < nwa; k += blockDim.x) {
    const size_t e = (size_t)p * nwa + k;
    KLS_UNLESS(SIM_IN(e, (int64_t)NR * pl), continue)
    const double sw = 0.5 * (f[k < nwa - 1 ? k + 1 : k] - f[k > 0 ? k - 1 : k]);
    const double dw = fabs(w1[e] - (f[k] + u * f[pl + k] + v * f[2 * pl + k]));
    const double dp = fabs(pha[e] - (f[3 * pl + k] + u * f[4 * pl + k] + v * f[5 * pl + k]));
    const double dr = fabs(ra[e] / (rc[iR] * f[6 * pl + k]) - 1.0);
    a += fabs(sw) * dw;
    b += fabs(sw) * (m * (dp + dq * fabs(f[k]) + q * dw) + (amax + 0.5) * dr);
  }
  for (int off = 16; off; off >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
  }
  __shared__ double2 sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_double2(a, b);
  __syncthreads();
  if (threadIdx.x) return;
  a = b = 0.0;
  for (int i = 0; i < (int)blockDim.x >> 5; ++i) { a += sh[i].x; b += sh[i].y; }
  out[p] = make_double2(a / KLS_PI, b / KLS_PI);
}

// samples of the 5 orbits a column is represented by: its mean, +- h along u, v
__global__ void reference_kernel(int Ne, int nwa, const double* __restrict__ fit,
                                 double* __restrict__ w1, double* __restrict__ ra,
                                 double* __restrict__ pha) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x, ie = blockIdx.y, q = blockIdx.z;
  if (k >= nwa) return;
  const size_t pl = (size_t)Ne * nwa, o = (size_t)ie * nwa + k;
  const double hu = q == 1 ? SIM_H : q == 2 ? -SIM_H : 0.0;
  const double hv = q == 3 ? SIM_H : q == 4 ? -SIM_H : 0.0;
  const size_t e = ((size_t)q * Ne + ie) * nwa + k;
  KLS_UNLESS(SIM_IN(e, 5 * pl) && SIM_IN(6 * pl + o, 7 * pl), return)
  w1[e] = fit[o] + hu * fit[pl + o] + hv * fit[2 * pl + o];
  pha[e] = fit[3 * pl + o] + hu * fit[4 * pl + o] + hv * fit[5 * pl + o];
  ra[e] = fit[6 * pl + o];
}

// What, D_u, D_v from the 5 tables [n_l][5 Ne][ldv]; per column the largest
// |What|, first and second differences and |l What_l|: size[ie][6] (the bits of
// a non-negative double order like the double)
__global__ void combine_kernel(int n_l, int Ne, int ldv, int l_min, const double* __restrict__ T,
                               double* __restrict__ V, float2* __restrict__ Vf,
                               float4* __restrict__ D, unsigned long long* __restrict__ size) {
  const int r = blockIdx.x, il = r / Ne, ie = r % Ne;
  double mx[6] = {0, 0, 0, 0, 0, 0};
  const double l = fabs((double)(l_min + il));
  for (int c = threadIdx.x; c < ldv; c += blockDim.x) {
    const size_t p = ((size_t)r * ldv + c) / 2;
    KLS_UNLESS(SIM_IN(((int64_t)il * 5 * Ne + 4 * Ne + ie) * ldv + c, (int64_t)n_l * 5 * Ne * ldv) &&
                   SIM_IN((int64_t)r * ldv + c, (int64_t)n_l * Ne * ldv), continue)
    double x[5];
    for (int q = 0; q < 5; ++q) x[q] = T[((size_t)il * 5 * Ne + q * Ne + ie) * ldv + c];
    const double du = (x[1] - x[2]) * (0.5 / SIM_H), dv = (x[3] - x[4]) * (0.5 / SIM_H);
    const double d2u = (x[1] + x[2] - 2.0 * x[0]) * (1.0 / (SIM_H * SIM_H));
    const double d2v = (x[3] + x[4] - 2.0 * x[0]) * (1.0 / (SIM_H * SIM_H));
    V[(size_t)r * ldv + c] = x[0];
    if (c & 1) { Vf[p].y = (float)x[0]; D[p].z = (float)du; D[p].w = (float)dv; }
    else { Vf[p].x = (float)x[0]; D[p].x = (float)du; D[p].y = (float)dv; }
    const double a[6] = {fabs(x[0]), fabs(du), fabs(dv), fabs(d2u), fabs(d2v), l * fabs(x[0])};
    for (int q = 0; q < 6; ++q) mx[q] = fmax(mx[q], a[q]);
  }
  for (int q = 0; q < 6; ++q) {
    for (int off = 16; off; off >>= 1)
      mx[q] = fmax(mx[q], __shfl_down_sync(0xffffffffu, mx[q], off));
    if ((threadIdx.x & 31) == 0)
      atomicMax(size + 6 * ie + q, (unsigned long long)__double_as_longlong(mx[q]));
  }
}

// The radii are uniform in ln Rc: ln Rc = mid + x h with x = 0, 1, .. (odd NR) or
// 1/2, 3/2, .. and their negatives.  Phi[0][k][d] = cos(d x_k h da), Phi[1] = sin;
// zero beyond the pairs and N_alpha.  d (x h da) is split into its rounded value
// and the rounding, which the first-order term restores.
__global__ void phase_kernel(int NR, int K2p, int Na, int Nap, double da,
                             const double* __restrict__ rc, double* __restrict__ Phi,
                             double2* __restrict__ rot) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (d >= Nap || k >= K2p) return;
  const double la = log(rc[0]), lb = log(rc[NR - 1]);
  auto phase = [&](double th, double* s, double* c) {
    const double t = d * th, e = fma((double)d, th, -t);
    double s0, c0;
    sincos(t, &s0, &c0);
    *c = fma(-e, s0, c0);
    *s = fma(e, c0, s0);
  };
  double s = 0.0, c = 0.0;
  if (d < Na && k < (NR + 1) / 2)
    phase(((NR & 1) ? (double)k : k + 0.5) * ((lb - la) / (double)(NR - 1)) * da, &s, &c);
  KLS_UNLESS(SIM_IN(((int64_t)K2p + k) * Nap + d, 2 * (int64_t)K2p * Nap), return)
  Phi[(size_t)k * Nap + d] = c;
  Phi[((size_t)K2p + k) * Nap + d] = s;
  if (k == 0) {
    phase(0.5 * (la + lb) * da, &s, &c);
    rot[d] = make_double2(c, s);
  }
}

// channel factors 1 / Rc, u / Rc, v / Rc of every orbit
__global__ void channel_kernel(int NR, int NPh, const double* __restrict__ rc,
                               const double* __restrict__ uv, double* __restrict__ U) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NPh) return;
  KLS_UNLESS(SIM_IN(2 * (int64_t)NPh + p, 3 * (int64_t)NPh), return)
  const double r = 1.0 / rc[p % NR];
  U[p] = r;
  U[NPh + p] = r * uv[p];
  U[2 * (size_t)NPh + p] = r * uv[NPh + p];
}

// ---- F ---------------------------------------------------------------------------
// With the mirrored radii mid +- x taken together, s = w+ + w-, t = w+ - w-,
//   C = sum s cos(d x h da), S = sum t sin(d x h da),
//   F(d) = A - i B,  (A, B) = (C, S) rotated by d da mid
// takes half the products of a sum over the radii: K = NR / 2 for the cosines
// with s and for the sines with t.  16 rows x 32 d per CTA, a warp 8 rows x 16 d:
// 2 column blocks x (cos, sin) x 3 channels x (re, im) = 24 DMMA blocks on 12 A
// fragments formed from the weights (18 FP64 operations a lane against 24 DMMA
// of 8 FMA a lane).  152 registers, 3 CTAs per SM: a warp of 32 d halves those
// operations but leaves 2 CTAs, 893 us against 817.  Bound: the FP64 pipe, which
// the DMMA and the weights' operations share (23 TFLOP/s of DMMA).  Default
// grid: 1370 -> 817 us per omega (before: a sum over all the radii).
constexpr int FA_R = 16, FA_D = 32, FA_K = 8, FA_STAGES = 3, FA_THREADS = 128;
constexpr int FA_S = 12;                  // row stride of w (16-byte values) and U (doubles)
constexpr int FA_PS = FA_D + 4;           // row stride of the phases, 4 mod 16
constexpr int FA_W = 0,                   // offsets in doubles: w+, w- [2][16][12] complex
              FA_U = FA_W + 2 * 2 * FA_R * FA_S,        // [3][2][16][12]
              FA_P = FA_U + 3 * 2 * FA_R * FA_S,        // [2][8][36]
              FA_STAGE = FA_P + 2 * FA_K * FA_PS;
constexpr size_t FA_SMEM = (size_t)FA_STAGES * FA_STAGE * sizeof(double);

__global__ void __launch_bounds__(FA_THREADS, 3)
fourier_kernel(int R, int Ne, int NR, int K2p, int Nap, int64_t K_pad,
               const double2* __restrict__ wt, const double* __restrict__ U,
               const double* __restrict__ Phi, const double2* __restrict__ rot,
               double4* __restrict__ F0, float4* __restrict__ Fc) {
  extern __shared__ __align__(16) double fsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int d0 = blockIdx.x * FA_D, r0 = blockIdx.y * FA_R, z = blockIdx.z;
  const double2* w = wt + (size_t)z * K_pad;
  const int nk = K2p / FA_K, up = NR >> 1, dn = (NR - 1) >> 1;   // R of pair 0, either side
  // a thread copies pair lk of row lr (weights and channel factors of both
  // sides) and 16 bytes of the cosines and of the sines
  const int lr = tid >> 3, lk = tid & 7, pk = tid >> 4, pc = tid & 15;
  const bool row_in = r0 + lr < R;
  const double2* wrow = w + (row_in ? (size_t)(r0 + lr) * NR : 0);
  const double* urow = U + (row_in ? (size_t)((r0 + lr) % Ne) * NR : 0);
  const size_t uch = (size_t)Ne * NR;
  const double* prow = Phi + (size_t)pk * Nap + d0 + 2 * pc;
  auto load = [&](int s, int kt) {
    double* st = fsm + (size_t)s * FA_STAGE;
    const int k = kt * FA_K + lk;
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const int iR = sd ? dn - k : up + k;
      const bool k_in = iR >= 0 && iR < NR;
      // (the centre of an odd grid is its own mirror: counted once)
      const bool u_in = k_in && !(sd && up == dn && k == 0);
      const int at = k_in ? iR : 0;
      KLS_IF(SIM_AT(wrow + at - w, K_pad))
      cp16z(st + FA_W + 2 * ((sd * FA_R + lr) * FA_S + lk), wrow + at, k_in && row_in ? 16 : 0);
#pragma unroll
      for (int ch = 0; ch < 3; ++ch)
        KLS_IF(SIM_AT(urow + ch * uch + at - U, 3 * uch))
        cp8z(st + FA_U + ((ch * 2 + sd) * FA_R + lr) * FA_S + lk, urow + ch * uch + at,
             u_in && row_in ? 8 : 0);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      KLS_IF(SIM_AT(prow + ((size_t)h * K2p + (size_t)kt * FA_K) * Nap + 1 - Phi,
                    2 * (int64_t)K2p * Nap))
      cp16z(st + FA_P + (h * FA_K + pk) * FA_PS + 2 * pc,
            prow + ((size_t)h * K2p + (size_t)kt * FA_K) * Nap, 16);
  };
  double c[3][2][2][2][2];                               // channel, (C, S), (re, im), block
#pragma unroll
  for (int h = 0; h < 3; ++h)
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int j = 0; j < 2; ++j) c[h][p][x][j][0] = c[h][p][x][j][1] = 0.0;
  const int wr = (warp & 1) * 8 + g, wc = (warp >> 1) * 16;
#pragma unroll
  for (int s = 0; s < FA_STAGES - 1; ++s) {
    if (s < nk) load(s, s);
    cp_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<FA_STAGES - 2>();
    __syncthreads();
    const int nxt = kt + FA_STAGES - 1;
    if (nxt < nk) load(nxt % FA_STAGES, nxt);
    cp_commit();
    const double* st = fsm + (size_t)(kt % FA_STAGES) * FA_STAGE;
#pragma unroll
    for (int kk = 0; kk < FA_K; kk += 4) {
      const int k = kk + t;
      const double2 xp = *reinterpret_cast<const double2*>(st + FA_W + 2 * (wr * FA_S + k));
      const double2 xm =
          *reinterpret_cast<const double2*>(st + FA_W + 2 * ((FA_R + wr) * FA_S + k));
      double bc[2], bs[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        bc[j] = st[FA_P + k * FA_PS + wc + 8 * j + g];
        bs[j] = st[FA_P + (FA_K + k) * FA_PS + wc + 8 * j + g];
      }
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const double mp = st[FA_U + (2 * h * FA_R + wr) * FA_S + k];
        const double mm = st[FA_U + ((2 * h + 1) * FA_R + wr) * FA_S + k];
        const double px = mm * xm.x, py = mm * xm.y;
        const double sx = fma(mp, xp.x, px), sy = fma(mp, xp.y, py);
        const double tx = fma(mp, xp.x, -px), ty = fma(mp, xp.y, -py);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dmma(c[h][0][0][j][0], c[h][0][0][j][1], sx, bc[j]);
          dmma(c[h][0][1][j][0], c[h][0][1][j][1], sy, bc[j]);
          dmma(c[h][1][0][j][0], c[h][1][0][j][1], tx, bs[j]);
          dmma(c[h][1][1][j][0], c[h][1][1][j][1], ty, bs[j]);
        }
      }
    }
  }
  cp_wait<0>();
  const int r = r0 + wr;
  if (r >= R) return;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int d = d0 + wc + 8 * j + 2 * t + x;
      KLS_UNLESS(SIM_AT(d, Nap), continue)
      const double2 q = rot[d];
      double a[3][4];                                    // A re, im, B re, im
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const double cr = c[h][0][0][j][x], ci = c[h][0][1][j][x];
        const double sr = c[h][1][0][j][x], si = c[h][1][1][j][x];
        a[h][0] = q.x * cr - q.y * sr;
        a[h][1] = q.x * ci - q.y * si;
        a[h][2] = q.y * cr + q.x * sr;
        a[h][3] = q.y * ci + q.x * si;
      }
      const size_t o = ((size_t)z * R + r) * Nap + d;
      KLS_UNLESS(SIM_AT(o, (int64_t)gridDim.z * R * Nap), continue)
      F0[o] = make_double4(a[0][0], a[0][1], a[0][2], a[0][3]);
      Fc[2 * o] = make_float4((float)a[1][0], (float)a[2][0], (float)a[1][1], (float)a[2][1]);
      Fc[2 * o + 1] = make_float4((float)a[1][2], (float)a[2][2], (float)a[1][3], (float)a[2][3]);
    }
}

// ---- the sum over (l, e) -------------------------------------------------------------
// For alphas i >= j with P = What_i conj(What_j), d = i - j, F(+-d) = A -+ i B:
//   X = sum A Re P + B Im P,  Y = sum A Im P - B Re P,
//   S[i, j] = X + i Y,  S[j, i] = X - i Y,
// and S[N-1-j, N-1-i] = S[i, j], so the pairs with i + j <= N - 1 are enough
// (a quarter of the matrix).  The channels add the same sums with
// Q = D_i conj(What_j) + What_i conj(D_j) in place of P: terms of at most
// SIM_FIRST of the others, summed in FP32 over a split's rows and added to the
// FP64 sums: the low part of a split whose error is 6e-14 of the sum.  Against 64-bit
// evaluations of 36 models over the range of grids M and the determinants are as far
// off as the table's (ratio of the errors 0.999 to 1.000).
//
// A CTA takes a tile of 32 x 32 pairs and a range of rows, either the FP64 sums
// or the FP32 ones (both kinds share the SMs, each on its own pipe); its two
// halves alternate rows, a thread has 4 x 4 pairs (i = ti + 8 q, j = tj + 8 p:
// the lanes of a quarter-warp read neighbouring d, and pairs with the same q - p
// share a d).  cp.async, 3 stages of 4 rows.  Bound: latency at 2 CTAs per SM (the
// 4 x 4 sums fill the registers; 3 CTAs spill, 1.35 x the time): the FP64 CTAs
// alone take 425 us and the FP32 ones 560, against 200 us each for their pipes
// and for the shared-memory reads (22 and 26 bytes a pair and row).  Tiles at the
// edges of the triangle leave out their empty 8 x 8 blocks in code of their own
// (PairShape) and have the fewer row splits for it.  Default grid: 1542 -> 1055 us
// per omega (before: 4 x 2 pairs with both sums in one thread, 64 bytes a pair, 2.03
// waves) -> 965 with the edges (run-time branches around the blocks: 1030);
// N_alpha = 101, 1071 rows, batch of 16: 22 -> 19.
constexpr int PR_T = 32, PR_ROWS = 4, PR_STAGES = 3, PR_THREADS = 128;
constexpr int PR_FA = 0, PR_FB = 1024,                 // bytes in a row: F of 64 d
              PR_W = 2048,                             // 32 i, 32 j: What or D
              PR_WF = 3072, PR_ROW = 3584;             // What in FP32
constexpr size_t PR_SMEM = (size_t)PR_STAGES * PR_ROWS * PR_ROW;
constexpr int PR_SLOT = PR_T * PR_T;        // pairs of a partial tile (double4 each)

// The 8 x 8 blocks (q, p) of a tile that hold pairs with i >= j (diagonal tiles:
// q >= p) and i + j <= N - 1 (q + p <= lim; lim is even)
template <bool DIAG, int LIM>
struct PairShape {
  static constexpr bool diag = DIAG;
  static constexpr int lim = LIM;
};

// row splits of a tile of weight w where a whole tile has k
__host__ __device__ __forceinline__ int tile_splits(int k, int w) {
  const int n = (k * w + 8) >> 4;
  return n > 0 ? n : 1;
}

__device__ __forceinline__ int pair_index(int Na, int i) {
  const int np = (Na + 1) >> 1, c0 = Na - np;
  return i >= c0 ? i - c0 : np - 1 - i;
}

__global__ void __launch_bounds__(PR_THREADS, 2)
pair_kernel(int R, int Na, int Nap, int ldv, int splits, int n_tiles,
            const int4* __restrict__ tiles, const double* __restrict__ V,
            const float2* __restrict__ Vf, const float4* __restrict__ D,
            const double4* __restrict__ F0, const float4* __restrict__ Fc,
            double4* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char psm[];
  const int tid = threadIdx.x;
  KLS_UNLESS(SIM_AT(blockIdx.x, n_tiles), return)
  const int4 tl = tiles[blockIdx.x];
  const bool fp64 = !(blockIdx.y & 1);                   // the kinds alternate over the SMs
  const int split = blockIdx.y >> 1, z = blockIdx.z, ns = tile_splits(splits, tl.z);
  if (split >= ns) return;
  const int rb = (int)((int64_t)R * split / ns), re = (int)((int64_t)R * (split + 1) / ns);
  const int nst = (re - rb + PR_ROWS - 1) / PR_ROWS;
  const int i0 = tl.x * PR_T, j0 = tl.y * PR_T, dlo = i0 - j0 - PR_T;   // d of window entry 0
  // 32 bytes a (row, d) of either kind
  const double2* f = fp64 ? reinterpret_cast<const double2*>(F0 + (size_t)z * R * Nap)
                          : reinterpret_cast<const double2*>(Fc + (size_t)z * R * Nap * 2);

  auto load = [&](int s, int it) {
    unsigned char* st = psm + (size_t)s * PR_ROWS * PR_ROW;
#pragma unroll
    for (int q = 0; q < PR_ROWS; ++q) {                  // F of 64 d, its two halves apart
      const int r = rb + it * PR_ROWS + q, w = tid >> 1, x = tid & 1, d = dlo + w;
      const bool in = r < re && d >= 0;
      KLS_IF(SIM_AT(in ? 2 * ((int64_t)r * Nap + d) + x : 0, 2 * (int64_t)R * Nap))
      cp16z(st + q * PR_ROW + (x ? PR_FB : PR_FA) + w * 16,
            f + (in ? 2 * ((size_t)r * Nap + d) + x : 0), in ? 16 : 0);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {                        // 4 rows x (32 i + 32 j)
      const int row = 2 * q + (tid >> 6), a = tid & 63, r = rb + it * PR_ROWS + row;
      const int al = a < 32 ? i0 + a : j0 + a - 32;
      const bool in = r < re && al < Na;
      const size_t o = in ? (size_t)r * (ldv >> 1) + pair_index(Na, al) : 0;
      unsigned char* dst = st + row * PR_ROW + PR_W + a * 16;
      KLS_UNLESS(SIM_AT(o, (int64_t)R * (ldv >> 1)), continue)
      if (fp64) {
        cp16z(dst, V + 2 * o, in ? 16 : 0);
      } else {
        cp16z(dst, D + o, in ? 16 : 0);
        cp8z(st + row * PR_ROW + PR_WF + a * 8, Vf + o, in ? 8 : 0);
      }
    }
  };

  const int ti = tid & 7, tj = (tid >> 3) & 7, half = tid >> 6;
  const int c0 = Na - ((Na + 1) >> 1);
  bool neg[4];                                           // alpha_i < 0: conj
#pragma unroll
  for (int q = 0; q < 4; ++q) neg[q] = i0 + ti + 8 * q < c0;
  double4* sh = reinterpret_cast<double4*>(psm);
  double4* out = part + (((size_t)z * n_tiles + blockIdx.x) * 2 * splits + blockIdx.y) * PR_SLOT;

  // rows it of the pipeline: body(row) for this half's rows
  auto rows = [&](auto body) {
#pragma unroll
    for (int s = 0; s < PR_STAGES - 1; ++s) {
      if (s < nst) load(s, s);
      cp_commit();
    }
    for (int it = 0; it < nst; ++it) {
      cp_wait<PR_STAGES - 2>();
      __syncthreads();
      const int nxt = it + PR_STAGES - 1;
      if (nxt < nst) load(nxt % PR_STAGES, nxt);
      cp_commit();
#pragma unroll
      for (int rr = 0; rr < PR_ROWS; rr += 2)
        body(psm + ((size_t)(it % PR_STAGES) * PR_ROWS + rr + half) * PR_ROW);
    }
    cp_wait<0>();
    __syncthreads();
  };
  // the body for this tile's shape
  auto by_shape = [&](auto body) {
    auto run = [&](auto t) { rows([&](const unsigned char* row) { body(row, t); }); };
    if (tl.x != tl.y) {
      if (tl.w == 6) run(PairShape<false, 6>{});
      else if (tl.w == 4) run(PairShape<false, 4>{});
      else if (tl.w == 2) run(PairShape<false, 2>{});
      else run(PairShape<false, 0>{});
    } else {
      if (tl.w == 6) run(PairShape<true, 6>{});
      else if (tl.w == 4) run(PairShape<true, 4>{});
      else if (tl.w == 2) run(PairShape<true, 2>{});
      else run(PairShape<true, 0>{});
    }
  };
  // the other half's sums, then the partial: [j][i], the lanes' i contiguous
  auto finish = [&](auto value) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int p = 0; p < 4; ++p)
        if (half) sh[(tj + 8 * p) * PR_T + ti + 8 * q] = value(q, p);
    __syncthreads();
    if (half) return;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int e = (tj + 8 * p) * PR_T + ti + 8 * q;
        const double4 o = sh[e], v = value(q, p);
        KLS_UNLESS(SIM_AT(out + e - part, (int64_t)gridDim.z * n_tiles * 2 * splits * PR_SLOT), continue)
        out[e] = make_double4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
      }
  };

  if (fp64) {
    double2 X[4][4], Y[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int p = 0; p < 4; ++p) X[q][p] = Y[q][p] = make_double2(0.0, 0.0);
    auto body = [&](const unsigned char* row, auto t) {
      double2 wi[4], wj[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        wi[q] = *reinterpret_cast<const double2*>(row + PR_W + (ti + 8 * q) * 16);
        if (neg[q]) wi[q].y = -wi[q].y;
        // alpha_j <= 0 in every pair that counts, so conj(What_j) is the stored pair
        wj[q] = *reinterpret_cast<const double2*>(row + PR_W + (32 + tj + 8 * q) * 16);
      }
#pragma unroll
      for (int dd = -3; dd < 4; ++dd) {
        if (dd < (t.diag ? 0 : -3) || dd > t.lim || -dd > t.lim) continue;
        const unsigned char* fd = row + (ti - tj + 8 * dd + PR_T) * 16;
        const double2 A = *reinterpret_cast<const double2*>(fd + PR_FA);
        const double2 B = *reinterpret_cast<const double2*>(fd + PR_FB);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int q = dd + p;
          if (q < 0 || q > 3) continue;
          if (q + p > t.lim) continue;
          const double pr = wi[q].x * wj[p].x - wi[q].y * wj[p].y;
          const double pi = wi[q].x * wj[p].y + wi[q].y * wj[p].x;
          X[q][p].x = fma(B.x, pi, fma(A.x, pr, X[q][p].x));
          X[q][p].y = fma(B.y, pi, fma(A.y, pr, X[q][p].y));
          Y[q][p].x = fma(-B.x, pr, fma(A.x, pi, Y[q][p].x));
          Y[q][p].y = fma(-B.y, pr, fma(A.y, pi, Y[q][p].y));
        }
      }
    };
    by_shape(body);
    finish([&](int q, int p) { return make_double4(X[q][p].x, X[q][p].y, Y[q][p].x, Y[q][p].y); });
    return;
  }
  // both channels in one packed FP32 operation: (u, v) in the two halves
  using kls_tc::f2_fma;
  using kls_tc::f2_mul;
  using kls_tc::f2_pack;
  uint64_t X[4][4][2], Y[4][4][2];                       // (re, im) x (u, v)
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 4; ++p) X[q][p][0] = X[q][p][1] = Y[q][p][0] = Y[q][p][1] = 0ull;
  const uint64_t minus = 0x8000000080000000ull;
  auto body = [&](const unsigned char* row, auto t) {
    uint64_t wr[4], wi[4], ni[4], dr[4], di[4];          // i: What, -Im What, D
    uint64_t vr[4], vi[4], nv[4], er[4], ei[4];          // j
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 w = *reinterpret_cast<const float2*>(row + PR_WF + (ti + 8 * q) * 8);
      const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(row + PR_W + (ti + 8 * q) * 16);
      const float im = neg[q] ? -w.y : w.y;
      wr[q] = f2_pack(w.x, w.x);
      wi[q] = f2_pack(im, im);
      ni[q] = wi[q] ^ minus;
      dr[q] = d.x;
      di[q] = neg[q] ? d.y ^ minus : d.y;
      const float2 v = *reinterpret_cast<const float2*>(row + PR_WF + (32 + tj + 8 * q) * 8);
      const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(row + PR_W + (32 + tj + 8 * q) * 16);
      vr[q] = f2_pack(v.x, v.x);
      vi[q] = f2_pack(v.y, v.y);
      nv[q] = vi[q] ^ minus;
      er[q] = e.x;
      ei[q] = e.y;
    }
#pragma unroll
    for (int dd = -3; dd < 4; ++dd) {
      if (dd < (t.diag ? 0 : -3) || dd > t.lim || -dd > t.lim) continue;
      const unsigned char* fd = row + (ti - tj + 8 * dd + PR_T) * 16;
      const ulonglong2 A = *reinterpret_cast<const ulonglong2*>(fd + PR_FA);
      const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(fd + PR_FB);
      const uint64_t nx = B.x ^ minus, ny = B.y ^ minus;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int q = dd + p;
        if (q < 0 || q > 3) continue;
        if (q + p > t.lim) continue;
        // Q = D_i conj(What_j) + What_i conj(D_j)
        const uint64_t qr = f2_fma(dr[q], vr[p], f2_fma(di[q], nv[p],
                                   f2_fma(wr[q], er[p], f2_mul(ni[q], ei[p]))));
        const uint64_t qi = f2_fma(dr[q], vi[p], f2_fma(di[q], vr[p],
                                   f2_fma(wr[q], ei[p], f2_mul(wi[q], er[p]))));
        X[q][p][0] = f2_fma(A.x, qr, f2_fma(B.x, qi, X[q][p][0]));
        X[q][p][1] = f2_fma(A.y, qr, f2_fma(B.y, qi, X[q][p][1]));
        Y[q][p][0] = f2_fma(A.x, qi, f2_fma(nx, qr, Y[q][p][0]));
        Y[q][p][1] = f2_fma(A.y, qi, f2_fma(ny, qr, Y[q][p][1]));
      }
    }
  };
  by_shape(body);
  auto sum = [](uint64_t v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
  };
  finish([&](int q, int p) {
    return make_double4(sum(X[q][p][0]), sum(X[q][p][1]), sum(Y[q][p][0]), sum(Y[q][p][1]));
  });
}

// 64 pairs of a tile per CTA, 4 threads per pair over every 4th split, added in
// order; a pair's up to 4 entries of I - M
__global__ void __launch_bounds__(256)
pair_reduce_kernel(int Na, int splits, int n_tiles, double G, const double* __restrict__ Nk,
                   const int4* __restrict__ tiles, const double4* __restrict__ part,
                   double2* __restrict__ Aall, double2* __restrict__ Mall) {
  __shared__ double4 sm[4][64];
  const int tile = blockIdx.x, e = blockIdx.y * 64 + (threadIdx.x & 63), sg = threadIdx.x >> 6;
  const int z = blockIdx.z;
  const int4 tl = tiles[tile];
  const double4* src = part + ((size_t)z * n_tiles + tile) * 2 * splits * PR_SLOT + e;
  const int slots = 2 * tile_splits(splits, tl.z);
  double4 s = make_double4(0, 0, 0, 0);
#pragma unroll 4
  for (int k = sg; k < slots; k += 4) {
    KLS_UNLESS(SIM_AT(src + (size_t)k * PR_SLOT - part,
                      (int64_t)gridDim.z * n_tiles * 2 * splits * PR_SLOT), continue)
    const double4 v = src[(size_t)k * PR_SLOT];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  sm[sg][threadIdx.x & 63] = s;
  __syncthreads();
  const int x = threadIdx.x & 63, o = threadIdx.x >> 6;
  const double4 a = sm[0][x], b = sm[1][x], c = sm[2][x], d = sm[3][x];
  const double Xr = ((a.x + b.x) + c.x) + d.x, Xi = ((a.y + b.y) + c.y) + d.y;
  const double Yr = ((a.z + b.z) + c.z) + d.z, Yi = ((a.w + b.w) + c.w) + d.w;
  const int i = tl.x * PR_T + (e & 31), j = tl.y * PR_T + (e >> 5);
  if (i < j || i + j > Na - 1) return;
  // o & 1: (j, i) instead of (i, j); o & 2: the mirrored entry
  if ((o & 1) && i == j) return;
  if ((o & 2) && i + j == Na - 1) return;
  const bool sw = o & 1;
  int row = sw ? j : i, col = sw ? i : j;
  const double sr = sw ? Xr + Yi : Xr - Yi, si = sw ? Xi - Yr : Xi + Yr;
  if (o & 2) { const int m = row; row = Na - 1 - col; col = Na - 1 - m; }
  const double n = Nk[col];
  const double mr = __dmul_rn(__dmul_rn(sr, G), n), mi = __dmul_rn(__dmul_rn(si, G), n);
  const size_t q = (size_t)row * Na + col;
  KLS_UNLESS(SIM_AT(q, (int64_t)Na * Na), return)
  Aall[(size_t)z * Na * Na + q] = make_double2((row == col ? 1.0 : 0.0) - mr, -mi);
  if (Mall && z == 0) Mall[q] = make_double2(mr, mi);
}

// eigenvectors of a symmetric n x n matrix (n <= SIM_PROBES) by cyclic Jacobi
// rotations; columns of E ordered by falling eigenvalue
void jacobi(double A[SIM_PROBES][SIM_PROBES], double E[SIM_PROBES][SIM_PROBES],
            double lam[SIM_PROBES]) {
  constexpr int n = SIM_PROBES;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) E[i][j] = i == j;
  for (int sweep = 0; sweep < 30; ++sweep) {
    double off = 0.0, tr = 0.0;
    for (int p = 0; p < n; ++p) {
      tr += A[p][p];
      for (int q = p + 1; q < n; ++q) off += std::fabs(A[p][q]);
    }
    if (!(off > 1e-17 * tr)) break;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) {
        if (A[p][q] == 0.0) continue;
        const double th = 0.5 * std::atan2(2.0 * A[p][q], A[q][q] - A[p][p]);
        const double c = std::cos(th), s = std::sin(th);
        for (int k = 0; k < n; ++k) {
          const double x = A[k][p], y = A[k][q];
          A[k][p] = c * x - s * y;
          A[k][q] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = A[p][k], y = A[q][k];
          A[p][k] = c * x - s * y;
          A[q][k] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = E[k][p], y = E[k][q];
          E[k][p] = c * x - s * y;
          E[k][q] = s * x + c * y;
        }
      }
  }
  for (int i = 0; i < n; ++i) lam[i] = A[i][i];
  for (int i = 0; i < n; ++i)
    for (int j = i + 1; j < n; ++j)
      if (lam[j] > lam[i]) {
        std::swap(lam[i], lam[j]);
        for (int k = 0; k < n; ++k) std::swap(E[k][i], E[k][j]);
      }
}

struct Scratch {                       // device arrays of the preparation
  KlsSlab slab;
  void* base = nullptr;
  ~Scratch() { cudaFree(base); }
};

// CTAs of the pair sum with k row splits of a whole tile
int pair_ctas(const kls_similar* s, int k) {
  int n = 0;
  for (int w : s->weight) n += 2 * tile_splits(k, w);
  return n;
}

constexpr int MAX_GRID_Y = 65535;

size_t f_bytes(const kls_similar* s) { return (size_t)s->R * s->Nap * 64; }

}  // namespace

void kls_similar_free(kls_ctx* c) {
  if (!c->sim) std::swap(c->sim, c->sim_off);
  kls_similar* s = c->sim;
  if (!s) return;
  cudaFree(s->slab);
  c->device_bytes -= (int64_t)s->slab_bytes;
  delete s;
  c->sim = nullptr;
}

// Reads the columns' common orbits off the samples and checks every orbit
// against them; leaves c->sim null when the model is not of this form.
int kls_similar_prepare(kls_ctx* c) {
  const int NR = c->NR, Ne = c->Ne, nwa = c->nwa, NPh = c->NPh;
  // fewer radii: the table's work is below this form's (2 N^2 NR against
  // 12 N NR + 22 N^2 per row)
  if (NR < 16 || nwa < 8) return KLS_OK;
  // beyond the grids of fourier_kernel, phase_kernel and fit_kernel: the table
  if ((int64_t)c->n_l * Ne > (int64_t)MAX_GRID_Y * FA_R || Ne > MAX_GRID_Y ||
      (NR + 1) / 2 > MAX_GRID_Y / FA_K * FA_K)
    return KLS_OK;
  Scratch sc;
  double *d_probe, *d_fit, *d_rfit, *d_ref, *d_of5, *d_T;
  double2* d_iv;
  int* d_ok;
  unsigned long long* d_mx;
  double2* d_mis;
  double* d_U = nullptr;
  const int PW = SIM_PROBES + 2;
  const size_t fitn = (size_t)Ne * nwa, n5 = (size_t)5 * Ne;
  const size_t tab = (size_t)c->n_l * Ne * c->ldv;
  sc.slab.add(&d_probe, (size_t)NPh * PW).add(&d_U, (size_t)2 * NPh).add(&d_fit, 7 * fitn);
  sc.slab.add(&d_rfit, (size_t)3 * Ne).add(&d_iv, Ne).add(&d_ref, 3 * n5 * nwa);
  sc.slab.add(&d_of5, (size_t)OF_COUNT * n5).add(&d_ok, n5).add(&d_T, 5 * tab);
  sc.slab.add(&d_mx, (size_t)6 * Ne).add(&d_mis, NPh);
  KLS_CK(c, sc.slab.alloc(&sc.base));
  probe_kernel<<<(NPh + 127) / 128, 128, 0, c->stream>>>(NPh, nwa, c->d_of, c->d_valid, c->d_w1,
                                                         c->d_pha, d_probe);
  KLS_LAUNCHED(c);
  std::vector<double> pr((size_t)NPh * PW), U((size_t)2 * NPh, 0.0), rfit((size_t)3 * Ne, 0.0);
  std::vector<double2> iv(Ne, make_double2(0.0, 0.0));
  std::vector<double> umax((size_t)2 * Ne, 0.0);
  std::vector<int> ok((size_t)5 * Ne, 0);
  KLS_CK(c, cudaMemcpyAsync(pr.data(), d_probe, pr.size() * sizeof(double),
                            cudaMemcpyDeviceToHost, c->stream));
  KLS_CK(c, cudaStreamSynchronize(c->stream));
  for (int ie = 0; ie < Ne; ++ie) {
    const double* col = pr.data() + (size_t)ie * NR * PW;
    const double* first = nullptr;
    double mean[SIM_PROBES + 1] = {0}, n = 0.0;
    for (int i = 0; i < NR; ++i) {
      const double* x = col + (size_t)i * PW;
      if (x[0] == 0.0) continue;
      if (!first) first = x;
      for (int q = 0; q <= SIM_PROBES; ++q) mean[q] += x[1 + q] - first[1 + q];
      n += 1.0;
    }
    if (!first) continue;
    for (int q = 0; q <= SIM_PROBES; ++q) mean[q] /= n;
    double A[SIM_PROBES][SIM_PROBES] = {{0}}, E[SIM_PROBES][SIM_PROBES], lam[SIM_PROBES];
    for (int i = 0; i < NR; ++i) {
      const double* x = col + (size_t)i * PW;
      if (x[0] == 0.0) continue;
      double d[SIM_PROBES];
      for (int q = 0; q < SIM_PROBES; ++q) d[q] = (x[2 + q] - first[2 + q]) - mean[1 + q];
      for (int a = 0; a < SIM_PROBES; ++a)
        for (int b = 0; b < SIM_PROBES; ++b) A[a][b] += d[a] * d[b];
    }
    jacobi(A, E, lam);
    double s2[2] = {0, 0}, sq[2] = {0, 0};
    for (int ch = 0; ch < 2; ++ch) {
      if (!(lam[ch] > 1e-28 * n)) continue;      // rounding of the samples themselves
      for (int i = 0; i < NR; ++i) {
        const double* x = col + (size_t)i * PW;
        if (x[0] == 0.0) continue;
        double u = 0.0;
        for (int q = 0; q < SIM_PROBES; ++q)
          u += E[q][ch] * ((x[2 + q] - first[2 + q]) - mean[1 + q]);
        U[(size_t)ch * NPh + (size_t)ie * NR + i] = u;
        s2[ch] += u * u;
        sq[ch] += u * (x[1] - first[1]);
        umax[2 * ie + ch] = std::max(umax[2 * ie + ch], std::fabs(u));
      }
    }
    iv[ie] = make_double2(s2[0] > 0 ? 1.0 / s2[0] : 0.0, s2[1] > 0 ? 1.0 / s2[1] : 0.0);
    rfit[3 * ie] = first[1] + mean[0];
    rfit[3 * ie + 1] = sq[0] * iv[ie].x;
    rfit[3 * ie + 2] = sq[1] * iv[ie].y;
    for (int q = 0; q < 5; ++q) ok[(size_t)q * Ne + ie] = 1;
  }
  std::vector<double> of5((size_t)OF_COUNT * n5, 0.0);
  for (int q = 0; q < 5; ++q)
    for (int ie = 0; ie < Ne; ++ie) {
      const double hu = q == 1 ? SIM_H : q == 2 ? -SIM_H : 0.0;
      const double hv = q == 3 ? SIM_H : q == 4 ? -SIM_H : 0.0;
      of5[(size_t)OF_OM1 * n5 + (size_t)q * Ne + ie] = 1.0;
      of5[(size_t)OF_OM2 * n5 + (size_t)q * Ne + ie] =
          rfit[3 * ie] + hu * rfit[3 * ie + 1] + hv * rfit[3 * ie + 2];
    }
  // a repeated precompute writes the same buffers again: a batch over models
  // (kls_multi.cu) holds their addresses
  kls_similar* s = c->sim ? c->sim : new kls_similar();
  c->sim = s;
  s->R = c->n_l * Ne;
  s->Nap = (c->Na + PR_T - 1) / PR_T * PR_T;
  s->K2p = ((NR + 1) / 2 + FA_K - 1) / FA_K * FA_K;
  std::vector<int4> tiles;
  s->weight.clear();
  for (int J = 0; 2 * J * PR_T <= c->Na - 1; ++J)
    for (int I = J; (I + J) * PR_T <= c->Na - 1; ++I) {
      const int lim = std::min(6, ((c->Na - 1 - (I + J) * PR_T) / 8 + 1) & ~1);
      int blocks = 0;
      for (int q = 0; q < 4; ++q)
        for (int p = 0; p < 4; ++p) blocks += q + p <= lim && (I > J || q >= p);
      // a row's operands cost about a quarter of a whole tile's time
      s->weight.push_back(4 + (3 * blocks + 3) / 4);
      tiles.push_back(make_int4(I, J, s->weight.back(), lim));
    }
  s->n_tiles = (int)tiles.size();
  auto bail = [&](int r) {
    kls_similar_free(c);
    return r;
  };
#define SIM_CK(call)                                                              \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) return bail(kls_cuda_fail(c, e_, #call));              \
  } while (0)
  if (!s->slab) {
    KlsSlab b;
    b.add(&s->V, tab).add(&s->Vf, tab / 2).add(&s->D, tab / 2).add(&s->U, (size_t)3 * NPh);
    b.add(&s->Phi, (size_t)2 * s->K2p * s->Nap).add(&s->rot, s->Nap).add(&s->tiles, tiles.size());
    SIM_CK(b.alloc(&s->slab));
    s->slab_bytes = b.bytes();
    c->device_bytes += (int64_t)s->slab_bytes;
  }
  SIM_CK(cudaMemcpyAsync(d_U, U.data(), U.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  SIM_CK(cudaMemcpyAsync(d_rfit, rfit.data(), rfit.size() * sizeof(double), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_iv, iv.data(), iv.size() * sizeof(double2), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_of5, of5.data(), of5.size() * sizeof(double), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_ok, ok.data(), ok.size() * sizeof(int), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(s->tiles, tiles.data(), tiles.size() * sizeof(int4),
                         cudaMemcpyHostToDevice, c->stream));
  SIM_CK(cudaMemsetAsync(d_mx, 0, (size_t)6 * Ne * sizeof(unsigned long long), c->stream));
  fit_kernel<<<dim3((nwa + 127) / 128, Ne), 128, 0, c->stream>>>(
      NR, Ne, nwa, d_probe, d_U, d_iv, c->d_rc, c->d_w1, c->d_ra, c->d_pha, d_fit);
  misfit_kernel<<<NPh, 256, 0, c->stream>>>(NR, Ne, nwa, std::abs(c->cfg.m), c->cfg.alpha_max,
                                            d_probe, d_U, d_rfit, c->d_rc, c->d_w1, c->d_ra,
                                            c->d_pha, d_fit, d_mis);
  double *rw = d_ref, *rr = rw + n5 * nwa, *rp = rr + n5 * nwa;
  reference_kernel<<<dim3((nwa + 127) / 128, Ne, 5), 128, 0, c->stream>>>(Ne, nwa, d_fit, rw, rr,
                                                                          rp);
  c->launches += 3;
  int r = kls_run_wl(c, (int)n5, 0, c->n_l, d_of5, d_ok, rw, rr, rp, d_T);
  if (r) return bail(r);
  combine_kernel<<<s->R, 128, 0, c->stream>>>(c->n_l, Ne, c->ldv, c->cfg.l_min, d_T, s->V, s->Vf,
                                                s->D, d_mx);
  const double da = c->Na > 1 ? (2.0 * c->cfg.alpha_max) / (double)(c->Na - 1) : 0.0;
  phase_kernel<<<dim3((s->Nap + 127) / 128, s->K2p), 128, 0, c->stream>>>(
      NR, s->K2p, c->Na, s->Nap, da, c->d_rc, s->Phi, s->rot);
  channel_kernel<<<(NPh + 127) / 128, 128, 0, c->stream>>>(NR, NPh, c->d_rc, d_U, s->U);
  c->launches += 3;
  SIM_CK(cudaGetLastError());
  std::vector<double> mx((size_t)6 * Ne);
  std::vector<double2> mis(NPh);
  SIM_CK(cudaMemcpyAsync(mx.data(), d_mx, mx.size() * sizeof(double), cudaMemcpyDeviceToHost,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(mis.data(), d_mis, mis.size() * sizeof(double2), cudaMemcpyDeviceToHost,
                         c->stream));
  SIM_CK(cudaStreamSynchronize(c->stream));
  bool fits = true;
  for (int ie = 0; ie < Ne && fits; ++ie) {
    const double* x = &mx[(size_t)6 * ie];
    // a phase l dw matters as far as What_l does
    const double leff = x[0] > 0.0 ? x[5] / x[0] : 0.0;
    double sum = 0.0, worst = 0.0, n = 0.0;
    for (int i = 0; i < NR; ++i) {
      const size_t p = (size_t)ie * NR + i;
      if (pr[p * PW] == 0.0) continue;
      const double e = leff * mis[p].x + mis[p].y;
      sum += e;
      n += 1.0;
      worst = std::max(worst, e);               // (a NaN stays in the sum)
    }
    fits = n == 0.0 || (sum <= n * SIM_FIT && worst <= SIM_WORST);
  }
  for (int ie = 0; ie < Ne && fits; ++ie) {
    const double *x = &mx[(size_t)6 * ie], u = umax[2 * ie], v = umax[2 * ie + 1];
    fits = u * x[1] + v * x[2] <= SIM_FIRST * x[0] &&
           (u * std::sqrt(x[3]) + v * std::sqrt(x[4])) *
                   (u * std::sqrt(x[3]) + v * std::sqrt(x[4])) <=
               2.0 * SIM_SECOND * x[0];
  }
  if (!fits) kls_similar_free(c);
  return KLS_OK;
#undef SIM_CK
}

// Row splits of a whole tile in the pair sum (the others have fewer, by weight),
// fixed per context; an FP64 and an FP32 CTA per tile and split, two of them on an
// SM at a time.  One wave while that leaves a split fewer than 64 rows, else up to 6
// waves (a last wave that is partly empty costs less of them).
int kls_similar_max_splits(const kls_ctx* c) {
  return std::max(1, std::min(c->sim->R / 8, MAX_GRID_Y / 2));   // (two kinds a split)
}
int kls_similar_splits(const kls_ctx* c) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  int s = 1, sum = 0;
  for (int w : c->sim->weight) sum += w;
  for (int waves = 1; waves <= 6; ++waves) {
    int k = std::max(1, sms * waves * 16 / sum);
    while (k > 1 && pair_ctas(c->sim, k) > 2 * sms * waves) --k;
    if (waves > 1 && c->sim->R < 64 * k) break;
    s = k;
  }
  return std::max(1, std::min(s, kls_similar_max_splits(c)));
}

// omegas whose F is held at once (256 MB, at least one), and its size
int kls_similar_chunk(const kls_ctx* c, int n) {
  return (int)std::max<size_t>(1, std::min<size_t>(n, ((size_t)256 << 20) / f_bytes(c->sim)));
}
size_t kls_similar_f_bytes(const kls_ctx* c, int n) {
  return f_bytes(c->sim) * kls_similar_chunk(c, n);
}
// omegas whose partials are held at once (1 GB, at least one), and their size in double2
// (a batch of 4096 omegas of N_alpha = 33 and 1071 rows: 71 GB of them)
int kls_similar_part_chunk(const kls_ctx* c, int n) {
  const size_t one = (size_t)c->sim->n_tiles * 2 * c->splits * PR_SLOT * sizeof(double4);
  return (int)std::max<size_t>(1, std::min<size_t>(n, ((size_t)1 << 30) / one));
}
size_t kls_similar_part_elems(const kls_ctx* c, int n) {
  return (size_t)kls_similar_part_chunk(c, n) * c->sim->n_tiles * 2 * c->splits * PR_SLOT * 2;
}
int kls_similar_ctas(const kls_ctx* c) { return pair_ctas(c->sim, c->splits); }

// F, pair sums and I - M of n omegas from their weights; no allocation, no
// synchronisation (capturable)
cudaError_t kls_similar_launch(const kls_ctx* c, cudaStream_t st, int n, const double2* wt,
                               void* F, double2* part, double2* A, double2* M, int* launches) {
  const kls_similar* s = c->sim;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(fourier_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)FA_SMEM)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)PR_SMEM)) != cudaSuccess)
    return e;
  const int nf = kls_similar_chunk(c, n), np = kls_similar_part_chunk(c, n);
  double4* F0 = reinterpret_cast<double4*>(F);
  float4* Fc = reinterpret_cast<float4*>(F0 + (size_t)nf * s->R * s->Nap);
  double4* p4 = reinterpret_cast<double4*>(part);
  const size_t slots = (size_t)s->n_tiles * 2 * c->splits * PR_SLOT;
  // ranges of omegas p0 .. p1 - 1 whose partials are reduced together
  for (int p0 = 0, p1; p0 < n; p0 = p1) {
    p1 = std::min(n, p0 + np);
    for (int b = p0; b < p1; b += nf) {
      const int m = std::min(nf, p1 - b);
      fourier_kernel<<<dim3(s->Nap / FA_D, (s->R + FA_R - 1) / FA_R, m), FA_THREADS, FA_SMEM, st>>>(
          s->R, c->Ne, c->NR, s->K2p, s->Nap, c->K_pad, wt + (size_t)b * c->K_pad, s->U, s->Phi,
          s->rot, F0, Fc);
      pair_kernel<<<dim3(s->n_tiles, 2 * c->splits, m), PR_THREADS, PR_SMEM, st>>>(
          s->R, c->Na, s->Nap, c->ldv, c->splits, s->n_tiles, s->tiles, s->V, s->Vf, s->D, F0, Fc,
          p4 + (b - p0) * slots);
      *launches += 2;
    }
    pair_reduce_kernel<<<dim3(s->n_tiles, PR_SLOT / 64, p1 - p0), 256, 0, st>>>(
        c->Na, c->splits, s->n_tiles, c->cfg.G, c->d_N, s->tiles, p4,
        A + (size_t)p0 * c->Na * c->Na, p0 ? nullptr : M);
    *launches += 1;
  }
  return cudaGetLastError();
}
