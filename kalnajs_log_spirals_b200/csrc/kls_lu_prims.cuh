// What both forms of the LU share: every kernel that inlines these rounds alike.
#pragma once
#include "kls_internal.cuh"

namespace {

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

}  // namespace
