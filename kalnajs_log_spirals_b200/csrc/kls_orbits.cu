// OrbitIntegration on the device: phase-space grid, per-orbit radial time
// integral (Omega_1), azimuthal phase integral (Omega_2), subsampled
// trajectory (w1, r, theta), Jacobian of (Rc, v) -> (E, L) and the
// Toomre-Zang distribution function with its E and L derivatives.
//
// Follows src/KalnajsLogSpiral/OrbitIntegration.jl:102-382 and
// src/KalnajsLogSpiral/Models.jl:40-169 of the reference.  One CTA per
// orbit; the reference's sequential cumsum over nw points
// (OrbitIntegration.jl:277-294) becomes a chunked block-wide prefix scan:
// each thread sums a contiguous chunk and leaves the chunk's running sums at its
// subsample points 1:nwai:nw; the chunk sums are scanned, and each thread adds
// its offset to the samples that it left.
//
// This translation unit is compiled without FMA contraction (-fmad=false)
// and keeps the reference's association order: v_r^2 = 2(E - ln x) x^2 - L^2
// cancels like 1/e^2 near the turning points of near-circular orbits, so a
// one-ulp change in any term moves Omega_1 by up to ~1e-10 relative.
#include "kls_internal.cuh"
#include <cmath>
#include <vector>

namespace {

constexpr int ORB_THREADS = 256;

struct OrbitParams {
  int NR, Ne, nw, nwa, nwai;
  double Rc_min, Rc_max, v_min;
  double L0, q1, qz, sigma_r0, DF_const;
  int n_zang;
  double dw;
  int quad_v;          // KLS_QUAD_* rule of the v grid (never DEFAULT here)
};

// trapezoid weight of point i of a sequence (OrbitIntegration.jl:63-74)
__host__ __device__ double trap_w(double xm, double x0, double xp, int i, int n) {
  if (n < 2) return 0.0;
  if (i == 0) return (xp - x0) / 2;
  if (i == n - 1) return (x0 - xm) / 2;
  return (xp - xm) / 2;
}

// Weight of point i of an n-point uniform grid x(.) under `rule`:
// KLS_QUAD_TRAPEZOID (OrbitIntegration.jl:63-74), KLS_QUAD_SIMPSON
// (OrbitIntegration.jl:79-95: the trapezoid rule for n < 3 or even n) or
// KLS_QUAD_BOOLE (2h/45 (7, 32, 12, 32, 14, ..., 7) for n = 4k + 1 >= 5,
// else the Simpson rule; NL_julia_boole.jl:186-217).
template <typename X>
__host__ __device__ double quad_w(int rule, const X& x, int i, int n) {
  auto trap = [&]() {
    double xm = i > 0 ? x(i - 1) : 0.0, xp = i < n - 1 ? x(i + 1) : 0.0;
    return trap_w(xm, x(i), xp, i, n);
  };
  if (rule == KLS_QUAD_TRAPEZOID) return trap();
  if (rule == KLS_QUAD_BOOLE && n >= 5 && (n - 1) % 4 == 0) {
    double dx = x(1) - x(0);
    double f = 2 * dx / 45;
    if (i == 0 || i == n - 1) return 7 * f;
    int r = i % 4;
    return r == 0 ? 14 * f : (r == 2 ? 12 * f : 32 * f);
  }
  if (n < 3 || (n % 2) == 0) return trap();
  double dx = x(1) - x(0);
  if (i == 0 || i == n - 1) return dx / 3;
  return (i % 2 == 1) ? 4 * dx / 3 : 2 * dx / 3;
}

// S_e weight of v point ie (OrbitIntegration.jl:119-123; Simpson unless the
// configuration selects another rule)
__device__ double v_weight(const OrbitParams& P, int ie) {
  auto v = [&](int i) { return kls_lin(P.v_min, 1.0, P.Ne, i); };
  return quad_w(P.quad_v, v, ie, P.Ne);
}

__device__ double taper(const OrbitParams& P, double L) {
  if (P.n_zang == 0) return 1.0;
  double La = fabs(L);
  if (La < 1e-12) return 0.0;
  return 1.0 / (1.0 + pow(P.L0 / La, (double)P.n_zang));
}

__device__ double df0(const OrbitParams& P, double E, double L) {
  double La = fabs(L);
  if (La < 1e-12) return 0.0;
  double s2 = P.sigma_r0 * P.sigma_r0;
  double r = P.DF_const * exp(-E / s2) * pow(La, P.qz) * taper(P, L);
  return isfinite(r) ? r : 0.0;
}

// Radial-integrand pieces at a point of the w grid, before the endpoints'
// extrapolation: x, sin w / v_r for the time, sin w / (v_r x) and the same over x
// for the phase.  `unit`: a power of two near 1 / Rc.
struct PointVals { double x, svr, svp, svpx; };

__device__ __forceinline__ PointVals point_vals(double rs, double drs, double E, double L2,
                                                bool nonradial, double unit, double cw,
                                                double sw) {
  PointVals v;
  v.x = rs - drs * cw;
  // v_r^2 cancels and keeps the reference's association order; what is made of it
  // does not: one reciprocal square root stands for its root and three divisions
  if (nonradial) {
    // (2 (E - V(x))) * x^2 - L^2
    const double vr2 = 2.0 * (E - log(v.x)) * (v.x * v.x) - L2, t = v.x * unit;
    const double q = sw * rsqrt(fmax(0.0, vr2) * (t * t));     // over x unit
    v.svpx = q * unit;
    v.svp = q * t;
    v.svr = v.svp * v.x;
  } else {
    double vr2 = 2.0 * (E - log(v.x));
    v.svr = sw * rsqrt(fmax(0.0, vr2));
    v.svp = v.svpx = 0.0;
  }
  return v;
}

// exclusive prefix sums of (a, b) over the block's threads, and the totals: sums
// in each warp, then every thread adds the warps before its own
__device__ void block_scan2(double& a, double& b, double2* sh, double2& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x = a, y = b;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double u = __shfl_up_sync(~0u, x, off), v = __shfl_up_sync(~0u, y, off);
    if (lane >= off) { x += u; y += v; }
  }
  if (lane == 31) sh[warp] = make_double2(x, y);
  x = __shfl_up_sync(~0u, x, 1);
  y = __shfl_up_sync(~0u, y, 1);
  if (lane == 0) x = y = 0.0;
  __syncthreads();
  double px = 0.0, py = 0.0;
  total = make_double2(0.0, 0.0);
  for (int w = 0; w < ORB_THREADS / 32; ++w) {
    if (w == warp) { px = total.x; py = total.y; }
    total.x += sh[w].x;
    total.y += sh[w].y;
  }
  a = px + x;
  b = py + y;
}

// cos and sin of the w grid in the order the orbit kernel reads them: step s of
// thread t's chunk at [s][t]
__global__ void order_kernel(int nw, int chunk, const double* __restrict__ cosw,
                             const double* __restrict__ sinw, double2* __restrict__ cs) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)(chunk + 1) * ORB_THREADS) return;
  const int64_t i = (e % ORB_THREADS) * chunk + e / ORB_THREADS;
  cs[e] = i < nw ? make_double2(cosw[i], sinw[i]) : make_double2(0.0, 0.0);
}

// table read, guarded in the bounds-checked build (plain t[i] otherwise)
#define ORB_TAB(t, i) KLS_LD(KLS_IB((i), P.nw, KS_ORBIT_TABLE), t[i], 0.0)
#define ORB_CS(p)                                                                       \
  KLS_LD(KLS_IB((p) - cs, (int64_t)(chunk + 1) * ORB_THREADS, KS_ORBIT_TABLE), *p,       \
         make_double2(0.0, 0.0))

// Bound: instruction issue (a logarithm and a reciprocal square root per point,
// about 190 instructions, 73 of them FP64).  80 registers and 24 warps per SM: 512
// threads at 64 registers take 16.7 ms, 256 at 64 16.4.  Default grid (25551 orbits
// of 100001 points): 59 -> 14.9 ms; before, every point was evaluated twice, with a
// root and three divisions, from tables that the lanes of a warp read a chunk apart.
__global__ void __launch_bounds__(ORB_THREADS, 3)
orbit_kernel(OrbitParams P, int chunk, const double* __restrict__ cosw, const double* __restrict__ sinw,
             const double2* __restrict__ cs,
             const double* __restrict__ rc_tab, const double* __restrict__ SRC,
             double* __restrict__ of, int NPh, int* __restrict__ valid,
             double* __restrict__ w1o, double* __restrict__ rao, double* __restrict__ phao) {
  __shared__ double2 sh_scan[ORB_THREADS / 32];
  __shared__ double sh_misc[4];
  const int p = blockIdx.x;
  const int iR = p % P.NR, ie = p / P.NR;
  const int tid = threadIdx.x;

  // ---- grid scalars (OrbitIntegration.jl:102-170), computed redundantly
  const double Rc = KLS_LD(KLS_IB(iR, P.NR, KS_ORBIT_TABLE), rc_tab[iR], 0.0);
  double v = kls_lin(P.v_min, 1.0, P.Ne, ie);
  if (fabs(v) < 1e-14) v = 1e-12;
  const double sg = (v > 0) ? 1.0 : ((v < 0) ? -1.0 : 0.0);
  const double ecc = 1.0 - fabs(v);
  const double R1 = Rc * (1.0 - ecc), R2 = Rc * (1.0 + ecc);
  double E;
  if (fabs(R2 * R2 - R1 * R1) > 1e-14) {
    E = (log(R2) * (R2 * R2) - log(R1) * (R1 * R1)) / (R2 * R2 - R1 * R1);
  } else {
    E = Rc * (1.0 / Rc) / 2 + log(Rc);
  }
  if (!isfinite(E)) E = log(R2);
  double L2 = 2.0 * (E - log(R2)) * (R2 * R2);
  if (L2 < 1e-14) L2 = 0.0;
  const double L = sqrt(L2) * sg;

  const double kap = sqrt(2.0) / Rc, Om = 1.0 / Rc;
  const int nw = P.nw, nwa = P.nwa, nwai = P.nwai;
  double* w1p = w1o + (size_t)p * nwa;
  double* rap = rao + (size_t)p * nwa;
  double* php = phao + (size_t)p * nwa;
  bool fin = true;
  double Om1 = 0.0, Om2 = 0.0;

  if (fabs(ecc) < 1e-10 || ecc < 0.01) {
    // circular (:222-229) and epicyclic (:232-241) branches
    Om1 = kap;
    Om2 = Om * sg;
    const bool circ = fabs(ecc) < 1e-10;
    const double a_j = (R2 - R1) / 2;
    for (int j = tid; j < nwa; j += blockDim.x) {
      int i = j * nwai;
      double wa = kls_lin(1e-8, KLS_PI - 1e-8, nw, i);
      double r, ph;
      if (circ) {
        r = Rc;
        ph = wa * Om2 / Om1;
      } else {
        r = Rc - a_j * ORB_TAB(cosw, i);
        ph = wa * Om2 / Om1 + 2 * Om / kap * a_j / Rc * ORB_TAB(sinw, i) * sg;
      }
      KLS_UNLESS(KLS_IB((int64_t)p * nwa + j, (int64_t)NPh * nwa, KS_ORBIT_SAMPLES), continue)
      w1p[j] = wa; rap[j] = r; php[j] = ph;
      fin = fin && isfinite(wa) && isfinite(r) && isfinite(ph);
    }
  } else {
    // general orbit (:244-302)
    const double rs = (R1 + R2) / 2, drs = (R2 - R1) / 2;
    const bool nonradial = L2 > 1e-12;
    const bool phase_int = (fabs(1.0 - ecc) > 1e-10) && nonradial;
    const double dtc = drs * P.dw;
    // svr / svr_phi with the reference's endpoint extrapolation
    // (NaN and infinity as from sin w / v_r: a product with an infinite q has x > 0)
    const double unit = exp2(-rint(log2(Rc)));
    auto vals_at = [&](int i, double cw, double sw, double& x, double& dt1, double& dt3) {
      PointVals a = point_vals(rs, drs, E, L2, nonradial, unit, cw, sw);
      x = a.x;
      if (i == 0 || i == nw - 1) {
        int i1 = (i == 0) ? 1 : nw - 2, i2 = (i == 0) ? 2 : nw - 3;
        PointVals b = point_vals(rs, drs, E, L2, nonradial, unit, ORB_TAB(cosw, i1),
                                 ORB_TAB(sinw, i1));
        PointVals c = point_vals(rs, drs, E, L2, nonradial, unit, ORB_TAB(cosw, i2),
                                 ORB_TAB(sinw, i2));
        if (i == nw - 1 || nonradial) a.svr = 2.0 * b.svr - c.svr;
        a.svpx = (2.0 * b.svp - c.svp) / x;
      }
      dt1 = dtc * a.svr;
      dt3 = dtc * a.svpx;
    };
    const int i0 = tid * chunk, i1 = min(nw, i0 + chunk);
    // the chunk's running sums of dt2 and dt4, left at its subsample points
    double st = 0.0, sp = 0.0;
    const int j0 = (i0 + nwai - 1) / nwai;
    auto mine = [&](int j) { return j < nwa && j * nwai < i1; };
    if (i0 < i1) {
      double x, dt1, dt3;
      double prev_t = 0.0, prev_p = 0.0;
      if (i0 > 0) vals_at(i0 - 1, ORB_TAB(cosw, i0 - 1), ORB_TAB(sinw, i0 - 1), x, prev_t, prev_p);
      int j = j0, next = j0 * nwai;
      const double2* src = cs + tid;
      double2 ahead = ORB_CS(src);                       // cs ends in a spare row
      for (int i = i0; i < i1; ++i) {
        const double2 q = ahead;
        src += ORB_THREADS;
        ahead = ORB_CS(src);
        vals_at(i, q.x, q.y, x, dt1, dt3);
        if (i > 0) { st += (prev_t + dt1) / 2; sp += (prev_p + dt3) / 2; }
        prev_t = dt1; prev_p = dt3;
        if (i == next && j < nwa) {
          KLS_IF(KLS_IB((int64_t)p * nwa + j, (int64_t)NPh * nwa, KS_ORBIT_SAMPLES)) {
            w1p[j] = st; rap[j] = x; php[j] = sp;
          }
          fin = fin && isfinite(x);
          ++j;
          next += nwai;
        }
      }
    }
    double2 tot;
    block_scan2(st, sp, sh_scan, tot);
    Om1 = KLS_PI / tot.x;
    // the thread's own samples: the chunks before it, then the units
    for (int j = j0; mine(j); ++j) {
      KLS_UNLESS(KLS_IB((int64_t)p * nwa + j, (int64_t)NPh * nwa, KS_ORBIT_SAMPLES), continue)
      const double wv = (st + w1p[j]) * Om1;
      double ph;
      if (phase_int) ph = L * (sp + php[j]);
      else ph = (j == 0) ? 0.0 : (KLS_PI / 2) * 1.0 * sg;
      w1p[j] = wv; php[j] = ph;
      fin = fin && isfinite(wv) && isfinite(ph);
      if (j == nwa - 1) sh_misc[0] = ph;
    }
    __syncthreads();
    Om2 = Om1 * sh_misc[0] / KLS_PI;
  }
  int all_fin = __syncthreads_and(fin ? 1 : 0);

  if (tid == 0) {
    // Jacobian (OrbitIntegration.jl:341-382)
    double jac = 0.0;
    if (fabs(R2 - R1) > 1e-12 && fabs(L) > 1e-12) {
      double V1 = log(R1), V2 = log(R2), dV1 = 1.0 / R1, dV2 = 1.0 / R2;
      double t1 = 2 * (E - V1) * R1 - dV1 * (R1 * R1);
      double t2 = 2 * (E - V2) * R2 - dV2 * (R2 * R2);
      double den = R2 * R2 - R1 * R1;
      double dj = fabs(t1 * t2 / den);
      jac = 2 * dj * Rc / Om1 / fabs(L);
    }
    if (fabs(L) <= 1e-12) {
      double DelE = 2.0 * (E - log(R1));
      jac = sqrt(fmax(DelE, 0.0)) * (1.0 / R2) * 2 * Rc / Om1;
      if (!isfinite(jac)) jac = 0.0;
    }
    // DF and derivatives (Models.jl:137-169), NaN -> 0 (:331-333)
    double F0 = df0(P, E, L);
    double FE = -F0 / (P.sigma_r0 * P.sigma_r0);
    double FL = 0.0;
    if (fabs(L) >= 1e-12) FL = F0 * (P.qz + P.n_zang - P.n_zang * taper(P, L)) / fabs(L);
    if (!isfinite(F0)) F0 = 0.0;
    if (!isfinite(FE)) FE = 0.0;
    if (!isfinite(FL)) FL = 0.0;
    // S_e quadrature weight (OrbitIntegration.jl:119-123); S_RC from the host
    double src = KLS_LD(KLS_IB(iR, P.NR, KS_ORBIT_TABLE), SRC[iR], 0.0);
    double se = v_weight(P, ie);
    double vals[OF_COUNT] = {Rc, ecc, v, R1, R2, E, L, L2, sg, se,
                             Om1, Om2, jac, F0, FE, FL, src * se * jac};
    for (int f = 0; f < OF_COUNT; ++f)
      KLS_IF(KLS_IB((int64_t)f * NPh + p, (int64_t)OF_COUNT * NPh, KS_ORBIT_FIELDS))
      of[(size_t)f * NPh + p] = vals[f];
    double ratio = Om2 / Om1;
    KLS_IF(KLS_IB(p, NPh, KS_ORBIT_FIELDS)) valid[p] = (all_fin && isfinite(ratio)) ? 1 : 0;
  }
}

}  // namespace

// Points of a thread's chunk: nw over the threads; up to a multiple of the
// subsampling where that is within 1 / 8, so that a warp's lanes leave their
// samples in the same step (default grid: 391 -> 400 points).
static int orbit_chunk(int nw, int nwai) {
  const int c = (nw + ORB_THREADS - 1) / ORB_THREADS, m = (c + nwai - 1) / nwai * nwai;
  return m - c <= c / 8 ? m : c;
}
size_t kls_orbit_table(int nw, int nwai) {
  return (size_t)(orbit_chunk(nw, nwai) + 1) * ORB_THREADS;
}

int kls_run_orbits(kls_ctx* c) {
  const kls_config& k = c->cfg;
  OrbitParams P{};
  P.NR = c->NR; P.Ne = c->Ne; P.nw = c->nw; P.nwa = c->nwa; P.nwai = c->nwai;
  P.Rc_min = k.Rc_min; P.Rc_max = k.Rc_max; P.v_min = k.v_min;
  P.L0 = k.L0; P.q1 = k.q1; P.qz = k.q1 - 1.0; P.n_zang = k.n_zang;
  P.sigma_r0 = 1.0 / std::sqrt(k.q1);
  // DF normalisation (Models.jl:53-54), Gamma of a real argument
  P.DF_const = 1.0 / (2.0 * KLS_PI * std::pow(2.0, P.qz / 2.0) * std::sqrt(KLS_PI) *
                      std::tgamma((P.qz + 1.0) / 2.0) * std::pow(P.sigma_r0, P.qz + 2.0));
  P.quad_v = k.quad_v == KLS_QUAD_DEFAULT ? KLS_QUAD_SIMPSON : k.quad_v;
  double w0 = kls_lin(1e-8, KLS_PI - 1e-8, c->nw, 0);
  double w1 = kls_lin(1e-8, KLS_PI - 1e-8, c->nw, 1);
  P.dw = w1 - w0;

  // Tables shared by every orbit, from the host C library: the w grid's cos
  // and sin, the log-spaced guiding-centre radii and their trapezoid weights
  // S_RC = Rc * trapz(ln Rc) (OrbitIntegration.jl:111-113, :188-193).  Near
  // a turning point x = rs - drs cos w cancels catastrophically, so the table
  // values, not just their accuracy, decide the last bits of Omega_1.
  std::vector<double> cw(c->nw), sw(c->nw), rc(c->NR), src(c->NR);
  for (int i = 0; i < c->nw; ++i) {
    double w = kls_lin(1e-8, KLS_PI - 1e-8, c->nw, i);
    cw[i] = std::cos(w);
    sw[i] = std::sin(w);
  }
  const double la = std::log10(k.Rc_min), lb = std::log10(k.Rc_max);
  for (int i = 0; i < c->NR; ++i) rc[i] = std::pow(10.0, kls_lin(la, lb, c->NR, i));
  {
    // S_RC = Rc * (weights on ln Rc): trapezoid unless configured
    std::vector<double> u(c->NR);
    for (int i = 0; i < c->NR; ++i) u[i] = std::log(rc[i]);
    const int rule = k.quad_rc == KLS_QUAD_DEFAULT ? KLS_QUAD_TRAPEZOID : k.quad_rc;
    auto x = [&](int i) { return u[i]; };
    for (int i = 0; i < c->NR; ++i) src[i] = rc[i] * quad_w(rule, x, i, c->NR);
  }
  KLS_CK(c, cudaMemcpyAsync(c->d_cosw, cw.data(), c->nw * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  KLS_CK(c, cudaMemcpyAsync(c->d_sinw, sw.data(), c->nw * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  KLS_CK(c, cudaMemcpyAsync(c->d_rc, rc.data(), c->NR * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  KLS_CK(c, cudaMemcpyAsync(c->d_SRC, src.data(), c->NR * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  const int chunk = orbit_chunk(c->nw, c->nwai);
  const int64_t ncs = (int64_t)kls_orbit_table(c->nw, c->nwai);
  kls_pre_mark(c, 0);
  order_kernel<<<(unsigned)((ncs + 255) / 256), 256, 0, c->stream>>>(
      c->nw, chunk, c->d_cosw, c->d_sinw, c->d_cs);
  KLS_LAUNCHED(c);
  orbit_kernel<<<c->NPh, ORB_THREADS, 0, c->stream>>>(P, chunk, c->d_cosw, c->d_sinw, c->d_cs, c->d_rc,
                                                      c->d_SRC, c->d_of, c->NPh, c->d_valid,
                                                      c->d_w1, c->d_ra, c->d_pha);
  KLS_LAUNCHED(c);
  kls_pre_mark(c, 1);
  // the host vectors must outlive the asynchronous copies
  KLS_CK(c, cudaStreamSynchronize(c->stream));
  return KLS_OK;
}

int kls_upload_alpha(kls_ctx* c) {
  // alpha grid and its weights (BasisFunctions.jl:106-107: trapezoid unless
  // configured)
  std::vector<double> a(c->Na), d(c->Na);
  for (int i = 0; i < c->Na; ++i) a[i] = kls_lin(-c->cfg.alpha_max, c->cfg.alpha_max, c->Na, i);
  const int rule =
      c->cfg.quad_alpha == KLS_QUAD_DEFAULT ? KLS_QUAD_TRAPEZOID : c->cfg.quad_alpha;
  auto x = [&](int i) { return a[i]; };
  for (int i = 0; i < c->Na; ++i) d[i] = quad_w(rule, x, i, c->Na);
  KLS_CK(c, cudaMemcpyAsync(c->d_alpha, a.data(), c->Na * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  KLS_CK(c, cudaMemcpyAsync(c->d_dalpha, d.data(), c->Na * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
  KLS_CK(c, cudaStreamSynchronize(c->stream));   // (a, d end here)
  return KLS_OK;
}
