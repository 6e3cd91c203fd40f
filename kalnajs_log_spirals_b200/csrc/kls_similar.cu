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
// Work per omega: 24 n_l Ne NR N_alpha flops in F and 28 FMA per pair and (l, e)
// row over N_alpha^2 / 4 pairs, against 2 N_alpha^2 n_l Ne NR for the table: at
// NR = 501, Ne = 51, N_alpha = 301, l = +-100 3.7e10 and 6.5e9 against 9.3e11.
#include "kls_internal.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

struct kls_similar {
  int R = 0;                  // rows (l, e): il * Ne + ie
  int Nap = 0;                // N_alpha padded to the pair tiles
  int NRp = 0;                // NR padded to the slabs of fourier_kernel
  double* V = nullptr;        // [R][ldv] What, pairs (Re, Im) at the alphas >= 0
  float* D = nullptr;         // [2][R][ldv] D_u, D_v
  double* U = nullptr;        // [2][Ne][NR] u, v
  double* Phi = nullptr;      // [NRp][2 Nap] cos, sin(d da ln Rc) / Rc
  int2* tiles = nullptr;      // pair tiles (I, J)
  int n_tiles = 0;
};

namespace {

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
  const double FE = of[(size_t)OF_FE * NPh + p], FL = of[(size_t)OF_FL * NPh + p];
  const double DJ = of[(size_t)OF_DJ * NPh + p];
  double* o = out + (size_t)p * (SIM_PROBES + 2);
  o[0] = valid[p] && !((FE == 0.0 && FL == 0.0) || DJ == 0.0) ? 1.0 : 0.0;
  o[1] = of[(size_t)OF_OM2 * NPh + p] / of[(size_t)OF_OM1 * NPh + p];
  for (int q = 0; q < 3; ++q) {
    const size_t k = (size_t)p * nwa + probe_at(nwa, q);
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
    const double w = w1[e], t = pha[e], u = U[p], v = U[(size_t)NR * Ne + p];
    if (n == 0.0) { w0 = w; p0 = t; }
    const double dw = w - w0, dp = t - p0;       // differences of near equals: exact
    sw += dw; sp += dp; sr += ra[e] / rc[iR]; n += 1.0;
    wu += dw * u; wv += dw * v; pu += dp * u; pv += dp * v;
  }
  const double2 iv = inv_var[ie];
  const size_t pl = (size_t)Ne * nwa, o = (size_t)ie * nwa + k;
  const double d = n > 0.0 ? 1.0 / n : 0.0;
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
  w1[e] = fit[o] + hu * fit[pl + o] + hv * fit[2 * pl + o];
  pha[e] = fit[3 * pl + o] + hu * fit[4 * pl + o] + hv * fit[5 * pl + o];
  ra[e] = fit[6 * pl + o];
}

// What, D_u, D_v from the 5 tables [n_l][5 Ne][ldv]; per column the largest
// |What|, first and second differences and |l What_l|: size[ie][6] (the bits of
// a non-negative double order like the double)
__global__ void combine_kernel(int n_l, int Ne, int ldv, int l_min, const double* __restrict__ T,
                               double* __restrict__ V, float* __restrict__ D,
                               unsigned long long* __restrict__ size) {
  const int r = blockIdx.x, il = r / Ne, ie = r % Ne;
  const size_t R = (size_t)n_l * Ne;
  double mx[6] = {0, 0, 0, 0, 0, 0};
  const double l = fabs((double)(l_min + il));
  for (int c = threadIdx.x; c < ldv; c += blockDim.x) {
    double x[5];
    for (int q = 0; q < 5; ++q) x[q] = T[((size_t)il * 5 * Ne + q * Ne + ie) * ldv + c];
    const double du = (x[1] - x[2]) * (0.5 / SIM_H), dv = (x[3] - x[4]) * (0.5 / SIM_H);
    const double d2u = (x[1] + x[2] - 2.0 * x[0]) * (1.0 / (SIM_H * SIM_H));
    const double d2v = (x[3] + x[4] - 2.0 * x[0]) * (1.0 / (SIM_H * SIM_H));
    const size_t o = (size_t)r * ldv + c;
    V[o] = x[0];
    D[o] = (float)du;
    D[R * ldv + o] = (float)dv;
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

// Phi[iR][2 d], [2 d + 1] = cos, sin(d da ln Rc) / Rc; zero beyond NR and N_alpha.
// d * (da ln Rc) is split into its rounded value and the rounding, which the
// first-order term restores.
__global__ void phase_kernel(int NR, int NRp, int Na, int Nap, double da,
                             const double* __restrict__ rc, double* __restrict__ Phi) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x, iR = blockIdx.y;
  if (d >= Nap || iR >= NRp) return;
  double s = 0.0, c = 0.0;
  if (d < Na && iR < NR) {
    const double th = da * log(rc[iR]), t = d * th, e = fma((double)d, th, -t);
    double s0, c0;
    sincos(t, &s0, &c0);
    c = fma(-e, s0, c0) / rc[iR];
    s = fma(e, c0, s0) / rc[iR];
  }
  *reinterpret_cast<double2*>(Phi + ((size_t)iR * Nap + d) * 2) = make_double2(c, s);
}

// ---- F ---------------------------------------------------------------------------
// F[r][d] = (A, B) = sum_R w(r, R) (cos, sin): 16 rows x 32 d per CTA, a warp 8
// rows x 16 d (4 column blocks) x 3 channels x (re, im) = 24 DMMA blocks; the
// channel weights are formed on the A fragment.  Bound: the DMMA pipe.
constexpr int FA_R = 16, FA_D = 32, FA_K = 16, FA_STAGES = 3, FA_THREADS = 128;
constexpr int FA_WS = 20;                 // row stride of w (16-byte values), 4 mod 8
constexpr int FA_US = 20;                 // row stride of u, v (doubles), 4 mod 16
constexpr int FA_PS = 2 * FA_D + 4;       // row stride of the phases, 4 mod 16
constexpr int FA_W = 0, FA_U = 2 * FA_R * FA_WS, FA_P = FA_U + 2 * FA_R * FA_US,
              FA_STAGE = FA_P + FA_K * FA_PS;   // offsets in doubles
constexpr size_t FA_SMEM = (size_t)FA_STAGES * FA_STAGE * sizeof(double);

__global__ void __launch_bounds__(FA_THREADS, 3)
fourier_kernel(int R, int Ne, int NR, int Nap, int64_t K_pad, const double2* __restrict__ wt,
               const double* __restrict__ U, const double* __restrict__ Phi,
               double4* __restrict__ F0, float4* __restrict__ Fc) {
  extern __shared__ __align__(16) double fsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int d0 = blockIdx.x * FA_D, r0 = blockIdx.y * FA_R, z = blockIdx.z;
  const double2* w = wt + (size_t)z * K_pad;
  const int nk = (NR + FA_K - 1) / FA_K;
  auto load = [&](int s, int kt) {
    double* st = fsm + (size_t)s * FA_STAGE;
    const int k0 = kt * FA_K;
#pragma unroll
    for (int q = 0; q < 2; ++q) {                        // w: 16 rows x 16 values
      const int e = tid + q * FA_THREADS, r = e >> 4, k = e & 15;
      const bool in = r0 + r < R && k0 + k < NR;
      cp16z(st + FA_W + 2 * (r * FA_WS + k),
            w + (in ? (size_t)(r0 + r) * NR + k0 + k : 0), in ? 16 : 0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {                        // u, v: 2 x 16 rows x 16
      const int e = tid + q * FA_THREADS, ch = e >> 8, r = (e >> 4) & 15, k = e & 15;
      const bool in = r0 + r < R && k0 + k < NR;
      cp8z(st + FA_U + (ch * FA_R + r) * FA_US + k,
           U + (in ? ((size_t)ch * Ne + (r0 + r) % Ne) * NR + k0 + k : 0), in ? 8 : 0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {                        // phases: 16 rows x 64
      const int e = tid + q * FA_THREADS, k = e >> 5, c = e & 31;
      cp16z(st + FA_P + k * FA_PS + 2 * c, Phi + ((size_t)(k0 + k) * Nap + d0 + c) * 2, 16);
    }
  };
  double c[3][2][4][2];                                  // channel, (re, im), block, (cos, sin)
#pragma unroll
  for (int h = 0; h < 3; ++h)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int j = 0; j < 4; ++j) c[h][x][j][0] = c[h][x][j][1] = 0.0;
  const int wr = (warp & 1) * 8, wc = (warp >> 1) * 32;
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
      const double2 x = *reinterpret_cast<const double2*>(st + FA_W + 2 * ((wr + g) * FA_WS + k));
      const double u = st[FA_U + (wr + g) * FA_US + k];
      const double v = st[FA_U + (FA_R + wr + g) * FA_US + k];
      const double a[3][2] = {{x.x, x.y}, {u * x.x, u * x.y}, {v * x.x, v * x.y}};
      double b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = st[FA_P + k * FA_PS + wc + 8 * j + g];
#pragma unroll
      for (int h = 0; h < 3; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dmma(c[h][0][j][0], c[h][0][j][1], a[h][0], b[j]);
          dmma(c[h][1][j][0], c[h][1][j][1], a[h][1], b[j]);
        }
    }
  }
  cp_wait<0>();
  const int r = r0 + wr + g;
  if (r >= R) return;
  const size_t row = ((size_t)z * R + r) * Nap + d0 + (wc >> 1);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const size_t o = row + 4 * j + t;
    F0[o] = make_double4(c[0][0][j][0], c[0][1][j][0], c[0][0][j][1], c[0][1][j][1]);
#pragma unroll
    for (int h = 1; h < 3; ++h)
      Fc[2 * o + h - 1] = make_float4((float)c[h][0][j][0], (float)c[h][1][j][0],
                                      (float)c[h][0][j][1], (float)c[h][1][j][1]);
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
// FP64 sums.
//
// A CTA takes a tile of 32 x 32 pairs and a range of rows; two halves of the
// CTA alternate rows, a thread has 4 x 2 pairs (i = ti + 8 q, j = tj + 8 q' +
// 16 h: the lanes of a quarter-warp read neighbouring d, and pairs with the
// same q - q' share a d).  cp.async, 3 stages of 4 rows.  Bound: issue slots
// and shared-memory reads about alike (12 FP64 + 32 FP32 FMA and 64 bytes a
// pair).
constexpr int PR_T = 32, PR_ROWS = 4, PR_STAGES = 3, PR_THREADS = 256;
constexpr int PR_FA = 0, PR_FB = 1024, PR_C1 = 2048, PR_C2 = 3072,   // bytes in a row: 64 d
              PR_WI = 4096, PR_WJ = 4608, PR_DI = 5120, PR_DJ = 5632, PR_ROW = 6144;
constexpr size_t PR_SMEM = (size_t)PR_STAGES * PR_ROWS * PR_ROW;
constexpr int PR_SLOT = PR_T * PR_T;        // pairs of a partial tile (double4 each)

__device__ __forceinline__ int pair_index(int Na, int i) {
  const int np = (Na + 1) >> 1, c0 = Na - np;
  return i >= c0 ? i - c0 : np - 1 - i;
}

__global__ void __launch_bounds__(PR_THREADS, 1)
pair_kernel(int R, int Na, int Nap, int ldv, int splits, int n_tiles,
            const int2* __restrict__ tiles, const double* __restrict__ V,
            const float* __restrict__ D, const double4* __restrict__ F0,
            const float4* __restrict__ Fc, double4* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char psm[];
  const int tid = threadIdx.x;
  const int2 tl = tiles[blockIdx.x];
  const int split = blockIdx.y, z = blockIdx.z;
  const int rb = (int)((int64_t)R * split / splits), re = (int)((int64_t)R * (split + 1) / splits);
  const int nst = (re - rb + PR_ROWS - 1) / PR_ROWS;
  const int i0 = tl.x * PR_T, j0 = tl.y * PR_T, dlo = i0 - j0 - PR_T;   // d of window entry 0
  const double4* f0 = F0 + (size_t)z * R * Nap;
  const float4* fc = Fc + (size_t)z * R * Nap * 2;

  auto load = [&](int s, int it) {
    unsigned char* st = psm + (size_t)s * PR_ROWS * PR_ROW;
#pragma unroll
    for (int q = 0; q < PR_ROWS; ++q) {                  // 256 values of 16 bytes: F of 64 d
      const int r = rb + it * PR_ROWS + q, w = tid >> 2, x = tid & 3, d = dlo + w;
      const bool in = r < re && d >= 0;
      const size_t o = in ? (size_t)r * Nap + d : 0;
      unsigned char* row = st + q * PR_ROW + w * 16;
      if (x < 2) cp16z(row + (x ? PR_FB : PR_FA), reinterpret_cast<const double2*>(f0 + o) + x,
                       in ? 16 : 0);
      else cp16z(row + (x == 2 ? PR_C1 : PR_C2), fc + 2 * o + (x - 2), in ? 16 : 0);
    }
    {                                                    // What: 4 rows x (32 i + 32 j)
      const int q = tid >> 6, a = tid & 63, r = rb + it * PR_ROWS + q;
      const int al = a < 32 ? i0 + a : j0 + a - 32;
      const bool in = r < re && al < Na;
      const size_t o = in ? (size_t)r * ldv + 2 * pair_index(Na, al) : 0;
      unsigned char* row = st + q * PR_ROW;
      cp16z(row + (a < 32 ? PR_WI + a * 16 : PR_WJ + (a - 32) * 16), V + o, in ? 16 : 0);
      unsigned char* dd = row + (a < 32 ? PR_DI + a * 16 : PR_DJ + (a - 32) * 16);
      cp8z(dd, D + o, in ? 8 : 0);
      cp8z(dd + 8, D + (in ? (size_t)R * ldv + o : 0), in ? 8 : 0);
    }
  };

  const int ti = tid & 7, tj = (tid >> 3) & 7, h = (tid >> 6) & 1, half = tid >> 7;
  const int c0 = Na - ((Na + 1) >> 1);
  double2 X[4][2], Y[4][2];
  float2 x32[4][2], y32[4][2];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      X[q][p] = Y[q][p] = make_double2(0.0, 0.0);
      x32[q][p] = y32[q][p] = make_float2(0.f, 0.f);
    }
  bool neg[4];                                           // alpha_i < 0: conj
#pragma unroll
  for (int q = 0; q < 4; ++q) neg[q] = i0 + ti + 8 * q < c0;

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
    for (int rr = 0; rr < PR_ROWS; rr += 2) {
      const unsigned char* row =
          psm + ((size_t)(it % PR_STAGES) * PR_ROWS + rr + half) * PR_ROW;
      double2 wi[4], wj[2];
      float4 di[4], dj[2];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        wi[q] = *reinterpret_cast<const double2*>(row + PR_WI + (ti + 8 * q) * 16);
        di[q] = *reinterpret_cast<const float4*>(row + PR_DI + (ti + 8 * q) * 16);
        if (neg[q]) { wi[q].y = -wi[q].y; di[q].y = -di[q].y; di[q].w = -di[q].w; }
      }
      // alpha_j <= 0 in every pair that counts, so conj(What_j) is the stored pair
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        wj[p] = *reinterpret_cast<const double2*>(row + PR_WJ + (tj + 8 * p + 16 * h) * 16);
        dj[p] = *reinterpret_cast<const float4*>(row + PR_DJ + (tj + 8 * p + 16 * h) * 16);
      }
#pragma unroll
      for (int dd = -1; dd < 4; ++dd) {
        const unsigned char* f = row + (ti - tj - 16 * h + 8 * dd + PR_T) * 16;
        const double2 A = *reinterpret_cast<const double2*>(f + PR_FA);
        const double2 B = *reinterpret_cast<const double2*>(f + PR_FB);
        const float4 u = *reinterpret_cast<const float4*>(f + PR_C1);
        const float4 v = *reinterpret_cast<const float4*>(f + PR_C2);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int q = dd + p;
          if (q < 0 || q > 3) continue;
          const double pr = wi[q].x * wj[p].x - wi[q].y * wj[p].y;
          const double pi = wi[q].x * wj[p].y + wi[q].y * wj[p].x;
          X[q][p].x = fma(B.x, pi, fma(A.x, pr, X[q][p].x));
          X[q][p].y = fma(B.y, pi, fma(A.y, pr, X[q][p].y));
          Y[q][p].x = fma(-B.x, pr, fma(A.x, pi, Y[q][p].x));
          Y[q][p].y = fma(-B.y, pr, fma(A.y, pi, Y[q][p].y));
          const float ar = (float)wi[q].x, ai = (float)wi[q].y;
          const float br = (float)wj[p].x, bi = (float)wj[p].y;
          const float ur = di[q].x * br - di[q].y * bi + (ar * dj[p].x - ai * dj[p].y);
          const float ui = di[q].x * bi + di[q].y * br + (ar * dj[p].y + ai * dj[p].x);
          const float vr = di[q].z * br - di[q].w * bi + (ar * dj[p].z - ai * dj[p].w);
          const float vi = di[q].z * bi + di[q].w * br + (ar * dj[p].w + ai * dj[p].z);
          float2 &x = x32[q][p], &y = y32[q][p];
          x.x += u.x * ur + u.z * ui + v.x * vr + v.z * vi;
          x.y += u.y * ur + u.w * ui + v.y * vr + v.w * vi;
          y.x += u.x * ui - u.z * ur + v.x * vi - v.z * vr;
          y.y += u.y * ui - u.w * ur + v.y * vi - v.w * vr;
        }
      }
    }
  }
  cp_wait<0>();
  __syncthreads();
  // rows of the other half, then the partial: [j][i], the lanes' i contiguous
  double4* sh = reinterpret_cast<double4*>(psm);
  double4* out = part + (((size_t)z * n_tiles + blockIdx.x) * splits + split) * PR_SLOT;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      X[q][p].x += x32[q][p].x; X[q][p].y += x32[q][p].y;
      Y[q][p].x += y32[q][p].x; Y[q][p].y += y32[q][p].y;
      const int e = (tj + 8 * p + 16 * h) * PR_T + ti + 8 * q;
      if (half) sh[e] = make_double4(X[q][p].x, X[q][p].y, Y[q][p].x, Y[q][p].y);
    }
  __syncthreads();
  if (half) return;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int e = (tj + 8 * p + 16 * h) * PR_T + ti + 8 * q;
      const double4 o = sh[e];
      out[e] = make_double4(X[q][p].x + o.x, X[q][p].y + o.y, Y[q][p].x + o.z, Y[q][p].y + o.w);
    }
}

// 64 pairs of a tile per CTA, 4 threads per pair over every 4th split, added in
// order; a pair's up to 4 entries of I - M
__global__ void __launch_bounds__(256)
pair_reduce_kernel(int Na, int splits, int n_tiles, double G, const double* __restrict__ Nk,
                   const int2* __restrict__ tiles, const double4* __restrict__ part,
                   double2* __restrict__ Aall, double2* __restrict__ Mall) {
  __shared__ double4 sm[4][64];
  const int tile = blockIdx.x, e = blockIdx.y * 64 + (threadIdx.x & 63), sg = threadIdx.x >> 6;
  const int z = blockIdx.z;
  const int2 tl = tiles[tile];
  const double4* src = part + ((size_t)z * n_tiles + tile) * splits * PR_SLOT + e;
  double4 s = make_double4(0, 0, 0, 0);
#pragma unroll 4
  for (int k = sg; k < splits; k += 4) {
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

struct Scratch {                       // device buffers of the preparation
  std::vector<void*> p;
  ~Scratch() {
    for (void* x : p) cudaFree(x);
  }
  template <typename T>
  cudaError_t get(T** out, size_t n) {
    cudaError_t e = cudaMalloc((void**)out, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) p.push_back(*out);
    return e;
  }
};

size_t f_bytes(const kls_similar* s) { return (size_t)s->R * s->Nap * 64; }

}  // namespace

void kls_similar_free(kls_ctx* c) {
  kls_similar* s = c->sim;
  if (!s) return;
  void* ptrs[] = {s->V, s->D, s->U, s->Phi, s->tiles};
  for (void* p : ptrs) cudaFree(p);
  delete s;
  c->sim = nullptr;
}

// Reads the columns' common orbits off the samples and checks every orbit
// against them; leaves c->sim null when the model is not of this form.
int kls_similar_prepare(kls_ctx* c) {
  const int NR = c->NR, Ne = c->Ne, nwa = c->nwa, NPh = c->NPh;
  // fewer radii: the table's work is below this form's (2 N^2 NR against
  // 24 N NR + 28 N^2 per row)
  if (NR < 16 || nwa < 8) return KLS_OK;
  Scratch sc;
  double *d_probe, *d_fit, *d_rfit, *d_ref, *d_of5, *d_T;
  double2* d_iv;
  int* d_ok;
  unsigned long long* d_mx;
  double2* d_mis;
  double* d_U = nullptr;
  const int PW = SIM_PROBES + 2;
  KLS_CK(c, sc.get(&d_probe, (size_t)NPh * PW));
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
  const size_t n5 = (size_t)5 * Ne;
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
  s->NRp = (NR + FA_K - 1) / FA_K * FA_K;
  const size_t fitn = (size_t)Ne * nwa, tab = (size_t)s->R * c->ldv;
  std::vector<int2> tiles;
  for (int J = 0; 2 * J * PR_T <= c->Na - 1; ++J)
    for (int I = J; (I + J) * PR_T <= c->Na - 1; ++I) tiles.push_back(make_int2(I, J));
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
  if (!s->V) {
    SIM_CK(cudaMalloc(&s->V, tab * sizeof(double)));
    SIM_CK(cudaMalloc(&s->D, 2 * tab * sizeof(float)));
    SIM_CK(cudaMalloc(&s->U, (size_t)2 * NPh * sizeof(double)));
    SIM_CK(cudaMalloc(&s->Phi, (size_t)s->NRp * s->Nap * 2 * sizeof(double)));
    SIM_CK(cudaMalloc(&s->tiles, tiles.size() * sizeof(int2)));
  }
  d_U = s->U;
  SIM_CK(sc.get(&d_fit, 7 * fitn));
  SIM_CK(sc.get(&d_rfit, rfit.size()));
  SIM_CK(sc.get(&d_iv, iv.size()));
  SIM_CK(sc.get(&d_ref, 3 * n5 * nwa));
  SIM_CK(sc.get(&d_of5, of5.size()));
  SIM_CK(sc.get(&d_ok, ok.size()));
  SIM_CK(sc.get(&d_T, 5 * tab));
  SIM_CK(sc.get(&d_mx, (size_t)6 * Ne));
  SIM_CK(sc.get(&d_mis, (size_t)NPh));
  SIM_CK(cudaMemcpyAsync(d_U, U.data(), U.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  SIM_CK(cudaMemcpyAsync(d_rfit, rfit.data(), rfit.size() * sizeof(double), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_iv, iv.data(), iv.size() * sizeof(double2), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_of5, of5.data(), of5.size() * sizeof(double), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(d_ok, ok.data(), ok.size() * sizeof(int), cudaMemcpyHostToDevice,
                         c->stream));
  SIM_CK(cudaMemcpyAsync(s->tiles, tiles.data(), tiles.size() * sizeof(int2),
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
  int r = kls_run_wl(c, (int)n5, c->cfg.l_min, c->n_l, d_of5, d_ok, rw, rr, rp, d_T);
  if (r) return bail(r);
  combine_kernel<<<s->R, 128, 0, c->stream>>>(c->n_l, Ne, c->ldv, c->cfg.l_min, d_T, s->V, s->D,
                                                d_mx);
  const double da = c->Na > 1 ? (2.0 * c->cfg.alpha_max) / (double)(c->Na - 1) : 0.0;
  phase_kernel<<<dim3((s->Nap + 127) / 128, s->NRp), 128, 0, c->stream>>>(
      NR, s->NRp, c->Na, s->Nap, da, c->d_rc, s->Phi);
  c->launches += 2;
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
      if (!(e <= worst)) worst = e;             // a NaN stays
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

// Row splits of the pair sum: about two CTAs per SM for one omega, at least 8
// rows each; fixed per context.
int kls_similar_max_splits(const kls_ctx* c) { return std::max(1, c->sim->R / 8); }
int kls_similar_splits(const kls_ctx* c) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  const int want = (2 * sms + c->sim->n_tiles - 1) / c->sim->n_tiles;
  return std::max(1, std::min(want, kls_similar_max_splits(c)));
}

// omegas whose F is held at once (256 MB, at least one), and its size
int kls_similar_chunk(const kls_ctx* c, int n) {
  return (int)std::max<size_t>(1, std::min<size_t>(n, ((size_t)256 << 20) / f_bytes(c->sim)));
}
size_t kls_similar_f_bytes(const kls_ctx* c, int n) {
  return f_bytes(c->sim) * kls_similar_chunk(c, n);
}
size_t kls_similar_part_elems(const kls_ctx* c, int n) {   // double2
  return (size_t)n * c->sim->n_tiles * c->splits * PR_SLOT * 2;
}
int kls_similar_ctas(const kls_ctx* c) { return c->sim->n_tiles * c->splits; }

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
  const int nf = kls_similar_chunk(c, n);
  double4* F0 = reinterpret_cast<double4*>(F);
  float4* Fc = reinterpret_cast<float4*>(F0 + (size_t)nf * s->R * s->Nap);
  double4* p4 = reinterpret_cast<double4*>(part);
  const size_t slots = (size_t)s->n_tiles * c->splits * PR_SLOT;
  for (int b = 0; b < n; b += nf) {
    const int m = std::min(nf, n - b);
    fourier_kernel<<<dim3(s->Nap / FA_D, (s->R + FA_R - 1) / FA_R, m), FA_THREADS, FA_SMEM, st>>>(
        s->R, c->Ne, c->NR, s->Nap, c->K_pad, wt + (size_t)b * c->K_pad, s->U, s->Phi, F0, Fc);
    pair_kernel<<<dim3(s->n_tiles, c->splits, m), PR_THREADS, PR_SMEM, st>>>(
        s->R, c->Na, s->Nap, c->ldv, c->splits, s->n_tiles, s->tiles, s->V, s->D, F0, Fc,
        p4 + b * slots);
    *launches += 2;
  }
  pair_reduce_kernel<<<dim3(s->n_tiles, PR_SLOT / 64, n), 256, 0, st>>>(
      c->Na, c->splits, s->n_tiles, c->cfg.G, c->d_N, s->tiles, p4, A, M);
  *launches += 1;
  return cudaGetLastError();
}
