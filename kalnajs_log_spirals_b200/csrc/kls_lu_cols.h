// The columns that one warp of the pipelined LU (kls_lu_pipe.cuh) owns, and the one that
// it factors next; and the batches that the pipelined form is the faster one for.  Plain
// C++ as well, so that both can be run on the host.
#pragma once
#ifdef __CUDACC__
#define LUP_HD __host__ __device__ __forceinline__
#else
#define LUP_HD inline
#endif

constexpr int LUP_WARPS = 8;

// 8 consecutive columns are on one CTA (its warps in turn), then on the next of the
// C: column (lp C + rank) 8 + warp is a warp's lp-th
struct LupCols {
  static constexpr int NONE = 0x7fffffff;      // (no column follows it: j + 1 is at most n)
  int first, step;
  int done = 0, left = 0, next, last = -1;     // factored, to come, the next one, the last one
  LUP_HD LupCols(int n, int C, int rank, int warp, int LP)
      : first(rank * LUP_WARPS + warp), step(C * LUP_WARPS) {
    for (int lp = 0; lp < LP; ++lp)
      if (col(lp) < n) { last = col(lp); ++left; }
    next = left ? first : NONE;
  }
  LUP_HD int col(int lp) const { return first + lp * step; }
  LUP_HD void taken() {                        // the next one is factored
    ++done;
    --left;
    next = left ? col(done) : NONE;
  }
};

// A wave of n matrices of N rows by one CTA each, us: the chain of a CTA, and for what
// 80 MB of the L2 do not hold the 32/3 N^3 bytes that reading and writing a matrix once a
// column makes, at 6.6 TB/s
inline double lu_cta_us(double n, double N) {
  const double out = n - 5e6 / (N * N);
  return n > 0 ? 1.35e-4 * N * N * N + 1.7 * N + (out > 0 ? 1.6e-6 * N * N * N * out : 0) : 0;
}
// Is the pipelined form the faster one for n matrices of N rows?  It takes a time per
// column (lup_classes) and wave of `clusters` matrices.  Measured from 41 to 512 rows and
// 1 to 1184 matrices: the choice is the faster form or at most 14% behind it.  One matrix
// is never near the line (97 against 296 us at N = 101, 552 against 4367 at 301); it is
// crossed at N = 101 between 64 matrices (240 against 299 us) and 96 (346 against 299), at
// 150 between 64 (618, 746) and 96 (1021, 748), at 301 never (1184: 59.2 against 67.6
// ms), at 400 between 48 (8.6, 12.2) and 148 (26.8, 22.7).
inline bool lup_wins(int n, int N, int clusters, double us_per_column, int sms) {
  const double pipe = (double)((n + clusters - 1) / clusters) * us_per_column * N;
  return pipe <= (double)(n / sms) * lu_cta_us(sms, N) + lu_cta_us(n % sms, N);
}
