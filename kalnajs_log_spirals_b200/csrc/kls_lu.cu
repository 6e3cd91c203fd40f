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
#include "kls_lu_pipe.h"
#include "kls_lu_prims.cuh"
#include <algorithm>
#include <cfloat>

namespace {

constexpr int LU_THREADS = 1024;

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

// ---- pipelined form (kls_lu_pipe.cuh) --------------------------------------------
// The size classes: rows per lane x columns per warp, CTAs per cluster.  4 columns
// a warp keep enough matrices on the device at once; a wider form (2 columns) for
// batches that it holds in one wave (7 matrices).  From <10,4> on, and a little in
// others, the registers do not hold all of it (160 bytes spilled a thread, <13,4> 1.0
// KB, <16,4> 2.1 KB).  1 matrix / 16, us:
//   N =  64  <2,2> x 4   51 /  52   (<2,8> x 1    71 /  71)
//   N = 101  <4,3> x 6   97 /  99   (<4,4> x 4   105 / 105, <4,2> x 8 128 / 249)
//   N = 192  <6,4> x 6  273 / 275   (<6,3> x 8   306 / 605), <6,2> x 12 236 / 700
//   N = 201  <7,5> x 6  344 / 348   (<7,4> x 8   333 / 656), <7,2> x 14 267 / 790
//   N = 256  <8,4> x 8  449 / 892   (<8,5> x 7   574 / 1140), <8,2> x 16 399 / 1185
//   N = 301 <10,4> x 10 550 / 1097  (<10,3> x 16 632 / 1887)
//   N = 400 <13,4> x 13 1249 / 3658 (<16,4> x 16 3277 / 9852)
//   N = 512 <16,4> x 16 2937 / 6513
// (in brackets: before the warp whose column is next polled)
struct LupClass {
  int n_max, C;
  LupKernels (*kernels)();
  double us;                  // a wave of matrices, per column (lup_wins)
  int Cw;                     // CTAs of the wider form
};
const LupClass lup_classes[] = {
    {64, 4, lup_kernels_64, 0.84, 0},     {128, 6, lup_kernels_128, 1.08, 0},
    {192, 6, lup_kernels_192, 1.41, 12},  {224, 6, lup_kernels_224, 1.71, 14},
    {256, 8, lup_kernels_256, 1.77, 16},  {320, 10, lup_kernels_320, 1.80, 0},
    {416, 13, lup_kernels_416, 2.90, 0},  {512, 16, lup_kernels_512, 4.00, 0},
};
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
        const LupKernels f = k.kernels();
        c->lu_full = lup_clusters(f.one, k.C, c->Na, false);
        c->lu_half = lup_clusters(f.one, k.C, c->Na, true);
        c->lu_wide = f.wide ? lup_clusters(f.wide, k.Cw, c->Na, false) : 0;
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
      KLS_CK(c, cudaLaunchKernelExC(&cfg, wide ? k.kernels().wide : k.kernels().one, args));
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
  return k >= 0 && lup_clusters(lup_classes[k].kernels().multi, lup_classes[k].C, n, false) ? k : -1;
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
  const void* fn = cls >= 0 ? lup_classes[cls].kernels().multi : nullptr;
  const int full = fn ? lup_clusters(fn, lup_classes[cls].C, max_Na, false) : 0;
  const bool half = n_pairs > full;
  const int clusters = full && half ? lup_clusters(fn, lup_classes[cls].C, max_Na, true) : full;
  if (full && lup_wins(n_pairs, max_Na, clusters, lup_classes[cls].us, lup_sms(device))) {
    const LupClass& k = lup_classes[cls];
    // one ring size for the class: as many slots as its largest matrix gets
    int slots = lup_slots(max_Na, half);
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = lup_config(k.C, n_pairs, lup_smem(max_Na, slots), st, &at);
    void* args[] = {&d_md, &d_pairs, (void*)&k.C, &slots, (void*)&wait};
    return (int)cudaLaunchKernelExC(&cfg, fn, args);
  }
  size_t sm = 2 * (size_t)max_Na * sizeof(double2);
  if (sm > 48 * 1024 &&
      (e = cudaFuncSetAttribute(multi_lu_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sm)) != cudaSuccess)
    return (int)e;
  multi_lu_kernel<<<n_pairs, LU_THREADS, sm, st>>>(d_md, d_pairs);
  return (int)cudaGetLastError();
}
