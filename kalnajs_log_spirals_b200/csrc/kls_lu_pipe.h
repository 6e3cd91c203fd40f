// Host side of the pipelined LU: its kernels by size class and their launch parameters.
#pragma once
#include "kls_internal.cuh"
#include "kls_lu_cols.h"

constexpr int LUP_THREADS = 32 * LUP_WARPS;

struct LupMeta {
  double2 u;                  // pivot
  int piv, pos;               // its row, and that row's position before the exchange
};

__host__ __device__ inline size_t lup_smem(int n, int slots) {
  return (size_t)slots * ((size_t)n * sizeof(double2) + sizeof(LupMeta) + sizeof(uint64_t)) + 16;
}

struct LupKernels {
  const void *one, *multi, *wide;        // (wide: fewer columns a warp, or null)
};
LupKernels lup_kernels_64();
LupKernels lup_kernels_128();
LupKernels lup_kernels_192();
LupKernels lup_kernels_224();
LupKernels lup_kernels_256();
LupKernels lup_kernels_320();
LupKernels lup_kernels_416();
LupKernels lup_kernels_512();
