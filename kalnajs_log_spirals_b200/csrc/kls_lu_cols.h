// The columns that one warp of the pipelined LU (kls_lu.cu) owns, and the one that
// it factors next.  Plain C++ as well, so that the schedule can be run on the host.
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
