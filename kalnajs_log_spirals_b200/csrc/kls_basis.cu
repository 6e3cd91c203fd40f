// BasisFunctions on the device.
//
// * W_l(alpha; J) table (BasisFunctions.jl:199-266, Eq. 41):
//     W[p, a, l] = (1/pi) sum_k Sw1_k cos(l w1_k + m phi_k) r_k^{-1/2} e^{-i alpha_a ln r_k}
//   evaluated per orbit as the product C[l,k] E[k,a] of a real matrix
//   C = Sw1_k cos(l w1_k + m phi_k) and a complex matrix
//   E = r_k^{-1/2} e^{-i alpha ln r_k}, on the FP64 tensor pipe (DMMA
//   m8n8k4).  C and E are generated in shared memory per 16-sample chunk:
//   each thread evaluates one anchor sincos and advances by complex rotation
//   over a short run (4 harmonics for C, 8 alphas for E); what depends on the
//   sample alone is computed once per 128 samples, one thread each.
//   Orbits with non-finite samples are zero rows (BasisFunctions.jl:224-226);
//   non-finite generated factors are zeroed (BasisFunctions.jl:248).
// * N_m(alpha) (BasisFunctions.jl:281-304, Eq. 46) through ln|Gamma(z)|:
//   Re[G(z1)G(z2)/(G(z3)G(z4))] = |G(z1)|^2/|G(z3)|^2 since z2 = conj(z1),
//   z4 = conj(z3).  ln|Gamma| uses Stirling's asymptotic series
//   (Bernoulli-number coefficients) after the upward recurrence
//   Gamma(z+1) = z Gamma(z) moves Re z above 15.
// * Per-row resonant data, row k = il*NPh + p (BasisFunctions.jl:127-153):
//   G_k = DJ_p * F0l[p,l], F0l = (l Om1 + m Om2) FE + m FL,
//   Omega_res = l Om1 + m Om2.
// * Resonant weights w_k(omega) = G_k / den for a batch of omegas, den = omega -
//   Omega_res, den := 1e-12 + 1e-12 i when |den| < 1e-12 (MatrixBuilder.jl:27-69).
//   Here and not with a contraction: every form takes them, and a module is loaded at
//   the first call that needs a kernel of it (this one by the precompute; the table
//   contraction's 3 MB took the first determinant of a process 1.5 ms).
#include "kls_internal.cuh"
#include <algorithm>
#include <cmath>
#include <cstdio>

namespace {

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// ---- W table kernel --------------------------------------------------------
constexpr int WL_AB = 64;      // alphas per CTA
constexpr int WL_BK = 16;      // samples per chunk
constexpr int WL_SC = WL_BK + 4;   // smem row stride of C [l][k] (== 4 mod 16)
constexpr int WL_SE = WL_AB + 4;   // smem row stride of E [k][a]
constexpr int WL_THREADS = 128;

struct WlParams {
  int NPh, nwa, np, ldv, n_l, l_min, m;   // np alphas >= 0
  int skip;              // first harmonics that are formed for their anchor's sake only
  double astep;          // alpha grid step
};

// orbit p's sample k, guarded in the bounds-checked build (plain t[k] otherwise)
#define WL_SMP(t, k) \
  KLS_LD(KLS_IB((int64_t)p * nwa + (k), (int64_t)NPh * nwa, KS_WL_SAMPLES), t[k], 0.0)

// Bound: the FP64 pipe, which DMMA and the generation of C and E share.  255 orbits
// of the default grid 4.61 -> 3.97 ms, all 25551 456 -> 395 ms: before, each of the 8
// threads of a sample computed its logarithm, root, two of its four sincos and its
// weight in every chunk.  MT tiles of 8 harmonics a CTA: 4, or 1 for up to 8 harmonics
// (one exported harmonic of 2121 orbits); a harmonic's bits are the same, as it is
// rotated from the same multiple of 4.
template <int MT>
__global__ void __launch_bounds__(WL_THREADS)
wl_kernel(WlParams P, const double* __restrict__ of, const int* __restrict__ valid,
          const double* __restrict__ w1g, const double* __restrict__ rag,
          const double* __restrict__ phag, const double* __restrict__ alpha,
          double* __restrict__ V) {
  constexpr int WL_LB = 8 * MT;   // harmonics per CTA
  __shared__ double sC[WL_LB * WL_SC];
  __shared__ double sEr[WL_BK * WL_SE];
  __shared__ double sEi[WL_BK * WL_SE];
  // per sample: w1, weight, m phi, cos and sin of w1, ln r, r^-1/2, cos and sin of
  // the alpha step
  __shared__ double smp[9][WL_THREADS];
  // one orbit's (l block, alpha block) CTAs are consecutive in launch order,
  // so its w1 / r / theta samples are read from DRAM once and then from L2
  const int nlb = (P.n_l + WL_LB - 1) / WL_LB, nab = (P.np + WL_AB - 1) / WL_AB;
  const int p = (int)(blockIdx.x / (unsigned)(nlb * nab));
  const int lb = (int)((blockIdx.x / (unsigned)nab) % (unsigned)nlb);
  const int ab = (int)(blockIdx.x % (unsigned)nab);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NPh = P.NPh, nwa = P.nwa;
  const double* w1 = w1g + (size_t)p * nwa;
  const double* ra = rag + (size_t)p * nwa;
  const double* pha = phag + (size_t)p * nwa;
  const bool ok = KLS_LD(KLS_IB(p, NPh, KS_WL_SAMPLES), valid[p] != 0, false);
  const double ratio = KLS_LD(KLS_IB(p, NPh, KS_WL_SAMPLES),
                              of[(size_t)OF_OM2 * NPh + p] / of[(size_t)OF_OM1 * NPh + p], 0.0);

  // accumulators: warp covers all harmonics (MT m-tiles) x 16 alphas (2 n-tiles)
  double accR[MT][2][2], accI[MT][2][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      accR[i][j][0] = accR[i][j][1] = 0.0;
      accI[i][j][0] = accI[i][j][1] = 0.0;
    }

  // generator assignment: 16 samples x 8 sub-runs
  const int gk = tid & 15, gsub = tid >> 4;       // gsub 0..7
  const int l_first = lb * WL_LB + gsub * 4;       // C: 4 harmonics (2 MT sub-runs)
  const int a_first = ab * WL_AB + gsub * 8;       // E: 8 alphas

  if (ok) {
    for (int k0 = 0; k0 < nwa; k0 += WL_BK) {
      if (k0 % WL_THREADS == 0 && k0 + tid < nwa) {
        const int k = k0 + tid;
        double wk = WL_SMP(w1, k), rk = WL_SMP(ra, k);
        double wm = k > 0 ? WL_SMP(w1, k - 1) : 0.0, wp = k < nwa - 1 ? WL_SMP(w1, k + 1) : 0.0;
        double sw;
        if (nwa < 2) sw = 0.0;
        else if (k == 0) sw = (wp - wk) / 2;
        else if (k == nwa - 1) sw = (wk - wm) / 2;
        else sw = (wp - wm) / 2;
        double phi = ratio * wk - WL_SMP(pha, k);
        double lr = log(rk), s, c;
        smp[0][tid] = wk;
        smp[1][tid] = sw;
        smp[2][tid] = (double)P.m * phi;
        sincos(wk, &s, &c);
        smp[3][tid] = c;
        smp[4][tid] = s;
        smp[5][tid] = lr;
        smp[6][tid] = 1.0 / sqrt(rk);
        sincos(-P.astep * lr, &s, &c);
        smp[7][tid] = c;
        smp[8][tid] = s;
      }
      if (k0 % WL_THREADS == 0) __syncthreads();
      // ---- generate C and E for samples k0..k0+15
      const int k = k0 + gk, e = k % WL_THREADS;
      if (k < nwa) {
        // C: cos(l w1 + m phi), anchor at l_first, rotate by w1
        double s, c, cs, ss;
        if (MT == 4 || gsub < 2 * MT) {
          const double sw = smp[1][e];
          double th = (double)(P.l_min + l_first) * smp[0][e] + smp[2][e];
          ss = smp[4][e];
          cs = smp[3][e];
          sincos(th, &s, &c);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            double v = sw * c;
            if (!isfinite(v)) v = 0.0;
            sC[(gsub * 4 + j) * WL_SC + gk] = (l_first + j < P.n_l) ? v : 0.0;
            double cn = c * cs - s * ss;
            s = s * cs + c * ss;
            c = cn;
          }
        }
        // E: r^{-1/2} e^{-i alpha ln r}, anchor at a_first, rotate by -astep ln r
        const double lr = smp[5][e], isq = smp[6][e];
        double ta = -KLS_LD(KLS_IB(min(a_first, P.np - 1), P.np, KS_WL_SAMPLES),
                            alpha[min(a_first, P.np - 1)], 0.0) * lr;
        sincos(ta, &s, &c);
        cs = smp[7][e];
        ss = smp[8][e];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          double er = c * isq, ei = s * isq;
          if (!(isfinite(er) && isfinite(ei))) { er = 0.0; ei = 0.0; }
          bool in = a_first + j < P.np;
          sEr[gk * WL_SE + gsub * 8 + j] = in ? er : 0.0;
          sEi[gk * WL_SE + gsub * 8 + j] = in ? ei : 0.0;
          double cn = c * cs - s * ss;
          s = s * cs + c * ss;
          c = cn;
        }
      } else {
        if (MT == 4 || gsub < 2 * MT)
#pragma unroll
          for (int j = 0; j < 4; ++j) sC[(gsub * 4 + j) * WL_SC + gk] = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          sEr[gk * WL_SE + gsub * 8 + j] = 0.0;
          sEi[gk * WL_SE + gsub * 8 + j] = 0.0;
        }
      }
      __syncthreads();
      // ---- 4 k-steps of m8n8k4
#pragma unroll
      for (int kk = 0; kk < WL_BK; kk += 4) {
        double a[MT], br[2], bi[2];
#pragma unroll
        for (int i = 0; i < MT; ++i) a[i] = sC[(i * 8 + (lane >> 2)) * WL_SC + kk + (lane & 3)];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          int col = warp * 16 + j * 8 + (lane >> 2);
          br[j] = sEr[(kk + (lane & 3)) * WL_SE + col];
          bi[j] = sEi[(kk + (lane & 3)) * WL_SE + col];
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            dmma(accR[i][j][0], accR[i][j][1], a[i], br[j]);
            dmma(accI[i][j][0], accI[i][j][1], a[i], bi[j]);
          }
      }
      __syncthreads();
    }
  }
  // ---- epilogue: W / pi into rows il*NPh + p
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    int il = lb * WL_LB + i * 8 + (lane >> 2);
    if (il < P.skip || il >= P.n_l) continue;
    size_t row = ((size_t)(il - P.skip) * NPh + p) * P.ldv;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      int a0 = ab * WL_AB + warp * 16 + j * 8 + 2 * (lane & 3);
      // alphas a0 and a0 + 1: columns 2 a0 .. 2 a0 + 3 (zero beyond np)
      if (2 * a0 >= P.ldv) continue;
      KLS_UNLESS(KLS_IB((int64_t)row + 2 * a0 + 1, (int64_t)P.n_l * NPh * P.ldv, KS_WL_OUT),
                 continue)
      *reinterpret_cast<double2*>(V + row + 2 * a0) =
          make_double2(accR[i][j][0] / KLS_PI, accI[i][j][0] / KLS_PI);
      if (2 * a0 + 2 >= P.ldv) continue;
      KLS_UNLESS(KLS_IB((int64_t)row + 2 * a0 + 3, (int64_t)P.n_l * NPh * P.ldv, KS_WL_OUT),
                 continue)
      *reinterpret_cast<double2*>(V + row + 2 * a0 + 2) =
          make_double2(accR[i][j][1] / KLS_PI, accI[i][j][1] / KLS_PI);
    }
  }
}

// ---- alpha grid and N_m(alpha) ------------------------------------------
// ln|Gamma(x + iy)| for x > 0 (Stirling series after upward recurrence).
__device__ double ln_abs_gamma(double x, double y) {
  double acc = 0.0;
  while (x < 15.0) {
    acc -= 0.5 * log(x * x + y * y);   // ln|z|
    x += 1.0;
  }
  // lnGamma(w) ~ (w - 1/2) ln w - w + ln(2 pi)/2 + sum_k c_k / w^(2k-1)
  double r = hypot(x, y), th = atan2(y, x);
  double lnr = log(r);
  double re = (x - 0.5) * lnr - y * th - x + 0.91893853320467274178;  // ln(2pi)/2
  // coefficients B_2k / (2k (2k-1)), k = 1..10
  const double cf[10] = {1.0 / 12.0,       -1.0 / 360.0,      1.0 / 1260.0,
                         -1.0 / 1680.0,    1.0 / 1188.0,      -691.0 / 360360.0,
                         1.0 / 156.0,      -3617.0 / 122400.0, 43867.0 / 244188.0,
                         -174611.0 / 125400.0};
  // 1/w = conj(w)/|w|^2 ; powers 1/w^(2k-1)
  double ir = x / (r * r), ii = -y / (r * r);            // 1/w
  double i2r = ir * ir - ii * ii, i2i = 2 * ir * ii;     // 1/w^2
  double pr = ir, pi = ii;
  for (int k = 0; k < 10; ++k) {
    re += cf[k] * pr;
    double nr = pr * i2r - pi * i2i;
    pi = pr * i2i + pi * i2r;
    pr = nr;
  }
  return re + acc;
}

// N_m(alpha) = |Gamma(z1)|^2 / |Gamma(z3)|^2 * pi * d_alpha,
// z1 = (m + 1/2 + i alpha)/2, z3 = (m + 3/2 + i alpha)/2
__global__ void n_kernel(int Na, int m, const double* __restrict__ alpha,
                         const double* __restrict__ dalpha, double* __restrict__ Nk) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Na) return;
  KLS_UNLESS(KLS_IB(i, Na, KS_NKERNEL), return)
  double a = alpha[i];
  double l1 = ln_abs_gamma((m + 0.5) / 2, a / 2);
  double l3 = ln_abs_gamma((m + 1.5) / 2, a / 2);
  Nk[i] = exp(2.0 * (l1 - l3)) * KLS_PI * dalpha[i];
}

__global__ void rows_kernel(int NPh, int n_l, int l_min, int m, int64_t K, int64_t K_pad,
                            const double* __restrict__ of, const int* __restrict__ valid,
                            double* __restrict__ Gk, double* __restrict__ Ok,
                            double* __restrict__ F0l) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K_pad) return;
  KLS_UNLESS(KLS_IB(k, K_pad, KS_ROWS), return)
  if (k >= K) { Gk[k] = 0.0; Ok[k] = 0.0; F0l[k] = 0.0; return; }
  int il = (int)(k / NPh), p = (int)(k % NPh);
  KLS_UNLESS(KLS_IB((int64_t)OF_DJ * NPh + p, (int64_t)OF_COUNT * NPh, KS_ROWS), return)
  double l = (double)(l_min + il);
  double om1 = of[(size_t)OF_OM1 * NPh + p], om2 = of[(size_t)OF_OM2 * NPh + p];
  double FE = of[(size_t)OF_FE * NPh + p], FL = of[(size_t)OF_FL * NPh + p];
  double DJ = of[(size_t)OF_DJ * NPh + p];
  double ores = l * om1 + m * om2;
  double f0l = ores * FE + m * FL;
  // an orbit with non-finite samples has W = 0: no weight either
  Gk[k] = KLS_LD(KLS_IB(p, NPh, KS_ROWS), valid[p], 0) ? DJ * f0l : 0.0 * (DJ * f0l);
  Ok[k] = ores;
  F0l[k] = f0l;
}

// ---- weights ---------------------------------------------------------------
// 1/z by Smith's algorithm (R. L. Smith, CACM 5(8), 1962), then a * (1/z):
// the same evaluation order as Julia's a / z for a real a.
__device__ __forceinline__ double2 real_over_complex(double a, double c, double d) {
  double p, q;
  if (fabs(d) <= fabs(c)) {
    double r = d / c;
    double t = 1.0 / (c + d * r);
    p = t;
    q = -r * t;
  } else {
    double r = c / d;
    double t = 1.0 / (d + c * r);
    p = r * t;
    q = -t;
  }
  return make_double2(a * p, a * q);
}

__device__ __forceinline__ double2 weight_at(double g, double ok, double wr, double wi) {
  double dr = wr - ok, di = wi;
  if (hypot(dr, di) < 1e-12) { dr = 1e-12; di = 1e-12; }
  return real_over_complex(g, dr, di);
}

__device__ __forceinline__ void weights_body(int64_t K_pad, double wr, double wi,
                                             const double* __restrict__ Gk,
                                             const double* __restrict__ Ok,
                                             double2* __restrict__ out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < K_pad;
       k += (int64_t)gridDim.x * blockDim.x)
    KLS_IF(KLS_IB(k, K_pad, KS_WEIGHTS)) out[k] = weight_at(Gk[k], Ok[k], wr, wi);
}

// anchored: w_k(omega) - w_k(omega_a), each with the denominator clamp; the
// FP64 difference loses ~|w| / |dw| ulps, far below the FP32 rounding the
// split-BF16 contraction applies next
__global__ void weights_kernel(int64_t K_pad, const double* __restrict__ omega,
                               const double* __restrict__ Gk, const double* __restrict__ Ok,
                               double2* __restrict__ wt, int anchored, double ar, double ai) {
  const int z = blockIdx.y;
  const double wr = omega[2 * z], wi = omega[2 * z + 1];
  double2* out = wt + (size_t)z * K_pad;
  if (!anchored) {
    weights_body(K_pad, wr, wi, Gk, Ok, out);
    return;
  }
  if (wr == ar && wi == ai) {                // at the anchor dM is exactly zero
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < K_pad;
         k += (int64_t)gridDim.x * blockDim.x)
      KLS_IF(KLS_IB(k, K_pad, KS_WEIGHTS)) out[k] = make_double2(0.0, 0.0);
    return;
  }
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < K_pad;
       k += (int64_t)gridDim.x * blockDim.x) {
    KLS_UNLESS(KLS_IB(k, K_pad, KS_WEIGHTS), continue)
    const double2 a = weight_at(Gk[k], Ok[k], wr, wi), b = weight_at(Gk[k], Ok[k], ar, ai);
    out[k] = make_double2(a.x - b.x, a.y - b.y);
  }
}

// one (model, omega) pair per grid row
__global__ void multi_weights_kernel(const kls_mdesc* __restrict__ md,
                                     const int2* __restrict__ pairs) {
  const int2 pz = pairs[blockIdx.y];
  const kls_mdesc& d = md[pz.x];
  const double* om = d.omega + 2 * pz.y;
  weights_body(d.K_pad, om[0], om[1], d.Gk, d.Ok, d.wt + (size_t)pz.y * d.K_pad);
}

}  // namespace

int kls_run_basis(kls_ctx* c) {
  const kls_config& k = c->cfg;
  int r = kls_upload_alpha(c);
  if (r) return r;
  n_kernel<<<(c->Na + 127) / 128, 128, 0, c->stream>>>(c->Na, k.m, c->d_alpha, c->d_dalpha,
                                                      c->d_N);
  KLS_LAUNCHED(c);
  rows_kernel<<<(unsigned)((c->K_pad + 255) / 256), 256, 0, c->stream>>>(
      c->NPh, c->n_l, k.l_min, k.m, c->K, c->K_pad, c->d_of, c->d_valid, c->d_Gk, c->d_Ok,
      c->d_F0l);
  KLS_LAUNCHED(c);
  return KLS_OK;
}

int kls_run_wl(kls_ctx* c, int n_orb, int il0, int n_l, const double* of, const int* valid,
               const double* w1, const double* ra, const double* pha, double* V) {
  WlParams P{};
  // harmonics are rotated from every 4th of the model's
  P.skip = il0 % 4;
  P.NPh = n_orb; P.nwa = c->nwa; P.np = (c->Na + 1) / 2; P.ldv = c->ldv; P.n_l = n_l + P.skip;
  P.l_min = c->cfg.l_min + il0 - P.skip; P.m = c->cfg.m;
  P.astep = c->Na > 1 ? (2.0 * c->cfg.alpha_max) / (double)(c->Na - 1) : 0.0;
  const int lb = P.n_l <= 8 ? 8 : 32;
  dim3 grid((unsigned)n_orb * ((P.n_l + lb - 1) / lb) * ((P.np + WL_AB - 1) / WL_AB));
  kls_pre_mark(c, 2);
  // the alphas >= 0 are the last np of the grid
  (lb == 8 ? wl_kernel<1> : wl_kernel<4>)<<<grid, WL_THREADS, 0, c->stream>>>(
      P, of, valid, w1, ra, pha, c->d_alpha + (c->Na - P.np), V);
  KLS_LAUNCHED(c);
  kls_pre_mark(c, 3);
  return KLS_OK;
}

int kls_build_table(kls_ctx* c) {
  const size_t n = (size_t)c->K_pad * c->ldv;
  const bool had = c->d_V != nullptr;
  cudaError_t e = c->d_V ? cudaSuccess : cudaMalloc(&c->d_V, n * sizeof(double));
  if (e != cudaSuccess) {
    cudaGetLastError();
    c->d_V = nullptr;
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    char buf[200];
    snprintf(buf, sizeof buf, "W table needs %.2f GB, device has %.2f GB free",
             n * sizeof(double) / 1e9, fr / 1e9);
    return kls_fail(c, KLS_ERR_OOM, buf);
  }
  c->device_bytes += had ? 0 : (int64_t)(n * sizeof(double));
  // zero the padding rows (K..K_pad-1)
  if (c->K_pad > c->K)
    KLS_CK(c, cudaMemsetAsync(c->d_V + (size_t)c->K * c->ldv, 0,
                              (size_t)(c->K_pad - c->K) * c->ldv * sizeof(double), c->stream));
  return kls_run_wl(c, c->NPh, 0, c->n_l, c->d_of, c->d_valid, c->d_w1, c->d_ra,
                    c->d_pha, c->d_V);
}

void kls_drop_table(kls_ctx* c) {
  if (!c->d_V) return;
  cudaFree(c->d_V);
  c->d_V = nullptr;
  c->device_bytes -= (int64_t)((size_t)c->K_pad * c->ldv * sizeof(double));
}

int kls_run_weights(kls_ctx* c, int n, const double* anchor) {
  int blocks = (int)std::min<int64_t>((c->K_pad + 255) / 256, 2048);
  weights_kernel<<<dim3(blocks, n), 256, 0, c->stream>>>(
      c->K_pad, c->d_omega, c->d_Gk, c->d_Ok, c->d_wt, anchor ? 1 : 0, anchor ? anchor[0] : 0.0,
      anchor ? anchor[1] : 0.0);
  KLS_LAUNCHED(c);
  return KLS_OK;
}

int kls_multi_launch_f64_weights(cudaStream_t st, const kls_mdesc* d_md, const int2* d_pairs,
                                 int n_pairs, int64_t max_K_pad) {
  int wblocks = (int)std::min<int64_t>((max_K_pad + 255) / 256, 1024);
  multi_weights_kernel<<<dim3(wblocks, n_pairs), 256, 0, st>>>(d_md, d_pairs);
  return (int)cudaGetLastError();
}
