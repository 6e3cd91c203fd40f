// Learned root proposer: a small MLP trained on the device by this file's own
// BF16 tensor-core kernels (no library GEMM).
//
//   features (5) -> [W1, b1, GELU] -> width -> ... -> [W_L, b_L] -> outputs (3)
//
// Parameters are FP32 masters (Adam moments FP32); every GEMM runs on BF16
// copies with FP32 accumulation (mma.sync m16n8k16 bf16 -> f32).  Each GEMM
// computes C[M x N] = A[M x K] * B[N x K]^T with both operands K-contiguous:
//   forward   Z_l  = H_{l-1} W_l^T + b_l        (A = H_{l-1}, B = W_l)
//   backward  dW_l = dZ_l^T H_{l-1}             (A = dZ_l^T, B = H_{l-1}^T)
//             dH   = dZ_l W_l                   (A = dZ_l,   B = W_l^T)
// so the epilogues also write transposed BF16 copies (H^T, dZ^T) and the
// update writes W and W^T in BF16.  GELU is the erf form
// 0.5 x (1 + erf(x / sqrt 2)).  The loss is the mean squared error over the
// batch and the outputs.
//
// A training step is 2 L + 1 launches for L layers: the forward layers (the first
// gathers and converts its rows of X, the last forms the loss and its gradient),
// dH of L - 1 layers, dW and the bias gradients of all layers in one, and the update.
// The steps of an epoch are queued without a wait; the losses are read at its end.
#include "kls_internal.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

struct kls_mlp;

namespace {

constexpr int ML_IN = 5, ML_OUT = 3;
constexpr int ML_ROWS = 1 << 22;      // rows of a training set kept on the device (48 B each)
constexpr int ML_PAD = 16;            // input / output dims padded to 16 for the MMA
constexpr int GT_THREADS = 128;
// the small and the large tile, rows = columns, with depth and stages of the
// cp.async pipeline; the number of row tiles of a batch follows from the small one
constexpr int GT_S = 32, GT_SK = 64, GT_L = 64, GT_LK = 32, GT_STAGES = 4;

// Sums of the columns [0, N) of S [rows][ld], each in the order of the rows
struct SumArgs {
  int rows, N, ld;
  const float* S;
  float* out;
};
constexpr int CS_ROWS = 64, CS_COLS = 32;        // a stage of a block's sums

enum Epi { EPI_STORE, EPI_GELU, EPI_OUT, EPI_MSE, EPI_GELU_BWD };

struct GemmArgs {
  int M, N, K;
  const __nv_bfloat16* A; int lda;     // A[m][k] at A[m * lda + k]
  const __nv_bfloat16* B; int ldb;     // B[n][k] at B[n * ldb + k]
  float* C; int ldc;                   // fp32 output (may be null)
  const float* bias;                   // [N]
  const float* Zin; int ldz;           // pre-activations for EPI_GELU_BWD
  __nv_bfloat16* H; int ldh;           // bf16 output [M][N] (may be null)
  __nv_bfloat16* Ht; int ldht;         // bf16 transposed output [N][ldht] (may be null)
  // the first layer: A is row idx[m] (m without idx) of X; its transpose to Xt
  const float* X;
  const int* idx;
  __nv_bfloat16* Xt;
  const float* T;                      // EPI_MSE: targets, by idx as X
  float* lpart;                        // EPI_MSE: sum of squares per row tile
};

__device__ __forceinline__ float gelu_f(float x) {
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_d(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) +
         x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm4(uint32_t* r, const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
// 16 bytes, of which the first `n` are read and the others zero
__device__ __forceinline__ void cp16n(void* smem, const void* gmem, int n) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
// the launches of a stream overlap their start with the end of the one before;
// nothing is read or written before that one is done
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;\ngriddepcontrol.wait;\n" ::: "memory");
}

// Column sums by a block: the block copies, CS_ROWS rows a stage, and the lanes of
// its first warp add.
__device__ void column_sums(const SumArgs& a, int blk, float* sm) {
  const int c0 = blk * CS_COLS, tid = threadIdx.x;
  auto load = [&](int s, int it) {
#pragma unroll
    for (int q = 0; q < CS_ROWS * CS_COLS / 4 / GT_THREADS; ++q) {
      const int e = q * GT_THREADS + tid, r = it * CS_ROWS + e / (CS_COLS / 4);
      const int c = e % (CS_COLS / 4) * 4;
      const bool in = r < a.rows && c0 + c < a.ld;
      cp16n(sm + (s * CS_ROWS + e / (CS_COLS / 4)) * CS_COLS + c,
            in ? a.S + (size_t)r * a.ld + c0 + c : a.S, in ? 16 : 0);
    }
  };
  const int n = (a.rows + CS_ROWS - 1) / CS_ROWS;
#pragma unroll
  for (int s = 0; s < GT_STAGES - 1; ++s) {
    if (s < n) load(s, s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  float s = 0.f;
  for (int it = 0; it < n; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GT_STAGES - 2));
    __syncthreads();
    if (it + GT_STAGES - 1 < n) load((it + GT_STAGES - 1) % GT_STAGES, it + GT_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    if (tid < 32) {
      const float* x = sm + it % GT_STAGES * CS_ROWS * CS_COLS + tid;
      const int m = min(CS_ROWS, a.rows - it * CS_ROWS);
      if (m == CS_ROWS) {
#pragma unroll 16
        for (int r = 0; r < CS_ROWS; ++r) s += x[r * CS_COLS];
      } else {
        for (int r = 0; r < m; ++r) s += x[r * CS_COLS];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (tid < 32 && c0 + tid < a.N) a.out[c0 + tid] = s;
}

// 4 warps on a BT x BT tile, 2 x 2; a stage holds BK of K for both operands, rows
// 16 bytes apart modulo 128 (ldmatrix without conflicts).  Every output adds its
// products over K in order, in steps of 16.
// Bound: latency - at a batch of 1024 and width 256 a GEMM has 0.13 Gflop and its
// operands are in L2, 5 to 11 us a launch.  A training step 850 -> 69 us, the
// forward pass of 820 rows 139 -> 42 us host to host; before: 2-byte loads, one
// stage, 64 x 64 tiles (16 blocks for dW), a thread per bias column, the batch
// gathered on the host and a wait per step.
template <int BT, int BK, int EPI>
__device__ __forceinline__ void gemm_tile(const GemmArgs& g, int blk,
                                          __nv_bfloat16 (*sm)[2][BT * (BK + 8)], float* sloss) {
  constexpr int LDS = BK + 8, MI = BT / 32, NJ = BT / 16, CH = BK / 8;
  constexpr int TLD = BT + 8;          // row stride of the transposed tile
  constexpr bool FIRST = EPI == EPI_GELU;              // (may be the layer that reads X)
  const int nx = (g.N + BT - 1) / BT;
  const int m0 = blk / nx * BT, n0 = blk % nx * BT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 1) * (BT / 2), wn = (warp & 1) * (BT / 2);
  const int gid = lane >> 2, tig = lane & 3;
  float acc[MI][NJ][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int t = 0; t < 4; ++t) acc[i][j][t] = 0.f;
  auto load = [&](int s, int it) {
#pragma unroll
    for (int q = 0; q < BT * CH / GT_THREADS; ++q) {
      const int e = q * GT_THREADS + tid, r = e / CH, k = e % CH * 8, gk = it * BK + k;
      const int kb = min(max(g.K - gk, 0), 8) * 2;       // rows may end inside the 16 bytes
      if (!(FIRST && g.X)) {
        const int n = m0 + r < g.M ? kb : 0;
        cp16n(&sm[s][0][r * LDS + k], n ? g.A + (size_t)(m0 + r) * g.lda + gk : g.A, n);
      }
      const int n = n0 + r < g.N ? kb : 0;
      cp16n(&sm[s][1][r * LDS + k], n ? g.B + (size_t)(n0 + r) * g.ldb + gk : g.B, n);
    }
  };
  const int nk = (g.K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < GT_STAGES - 1; ++s) {
    if (s < nk) load(s, s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  if (FIRST && g.X && tid < BT) {               // K = ML_PAD: one stage
    const int r = m0 + tid;
    const float* x = g.X + (size_t)(r < g.M ? (g.idx ? g.idx[r] : r) : 0) * ML_IN;
    __align__(16) __nv_bfloat16 v[ML_PAD];
#pragma unroll
    for (int c = 0; c < ML_PAD; ++c)
      v[c] = __float2bfloat16(c < ML_IN && r < g.M ? x[c < ML_IN ? c : 0] : 0.f);
#pragma unroll
    for (int c = 0; c < ML_PAD; c += 8)
      *reinterpret_cast<uint4*>(&sm[0][0][tid * LDS + c]) = *reinterpret_cast<const uint4*>(v + c);
    if (g.Xt && n0 == 0)
#pragma unroll
      for (int c = 0; c < ML_PAD; ++c) g.Xt[(size_t)c * g.ldht + r] = v[c];
  }
  // the epilogue's operands, fetched under the products
  const int cl = wn + 2 * tig, rl = wm + gid;            // in the tile, + 8 j and + 16 i
  float zin[MI][NJ][4];
  if (EPI == EPI_GELU_BWD) {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = m0 + rl + 16 * i + 8 * h, c = n0 + cl + 8 * j;
          float2 z = make_float2(0.f, 0.f);
          if (r < g.M && c < g.N) z = *reinterpret_cast<const float2*>(g.Zin + (size_t)r * g.ldz + c);
          zin[i][j][2 * h] = z.x;
          zin[i][j][2 * h + 1] = z.y;
        }
  }
  const int lr = lane & 7, lq = lane >> 3;
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GT_STAGES - 2));
    __syncthreads();
    if (it + GT_STAGES - 1 < nk) load((it + GT_STAGES - 1) % GT_STAGES, it + GT_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const __nv_bfloat16 *sA = sm[it % GT_STAGES][0], *sB = sm[it % GT_STAGES][1];
    const int kend = min(BK, g.K - it * BK);
#pragma unroll
    for (int ks = 0; ks < BK; ks += 16) {
      if (ks >= kend) break;
      uint32_t af[MI][4], bf[NJ][2];
#pragma unroll
      for (int i = 0; i < MI; ++i)     // rows 0-7, 8-15 of k 0-7, then of k 8-15
        ldsm4(af[i], sA + (wm + 16 * i + lr + 8 * (lq & 1)) * LDS + ks + 8 * (lq >> 1));
#pragma unroll
      for (int j = 0; j < NJ; j += 2)  // columns 8 j: k 0-7, 8-15, then columns 8 (j + 1)
        ldsm4(bf[j], sB + (wn + 8 * j + lr + 8 * (lq >> 1)) * LDS + ks + 8 * (lq & 1));
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma_bf16(acc[i][j], af[i], bf[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();

  // fragment element t at row gid (+ 8 for t >= 2), column 2 tig + (t & 1)
  __nv_bfloat16* tr = &sm[0][0][0];
  float loss = 0.f;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = m0 + rl + 16 * i + 8 * h, c = n0 + cl + 8 * j;
        float o[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const bool in = r < g.M && c + x < g.N;
          float v = acc[i][j][2 * h + x];
          if (EPI == EPI_STORE) {
            if (in) g.C[(size_t)r * g.ldc + c + x] = v;
          } else if (EPI == EPI_GELU_BWD) {
            v = v * gelu_d(zin[i][j][2 * h + x]);
            if (in) g.C[(size_t)r * g.ldc + c + x] = v;
          } else {
            v = in ? v + g.bias[c + x] : 0.f;
            if (EPI == EPI_OUT) {
              if (in && c + x < ML_OUT) g.C[(size_t)r * ML_OUT + c + x] = v;
            } else if (EPI == EPI_MSE) {
              float d = 0.f;
              if (in && c + x < ML_OUT)
                d = v - g.T[(size_t)(g.idx ? g.idx[r] : r) * ML_OUT + c + x];
              loss += d * d;
              v = 2.f * d / (float)(g.M * ML_OUT);
              if (in) g.C[(size_t)r * g.ldc + c + x] = v;
            } else {
              if (in && g.C) g.C[(size_t)r * g.ldc + c + x] = v;
              v = gelu_f(v);
            }
          }
          o[x] = v;
        }
        if (EPI == EPI_STORE || EPI == EPI_OUT) continue;
        const __nv_bfloat162 b = __floats2bfloat162_rn(o[0], o[1]);
        if (g.H && r < g.M && c < g.N)
          *reinterpret_cast<__nv_bfloat162*>(g.H + (size_t)r * g.ldh + c) = b;
        if (g.Ht) {
          tr[(cl + 8 * j) * TLD + rl + 16 * i + 8 * h] = b.x;
          tr[(cl + 8 * j + 1) * TLD + rl + 16 * i + 8 * h] = b.y;
        }
      }
  if (EPI == EPI_MSE) {
#pragma unroll
    for (int off = 16; off; off >>= 1) loss += __shfl_xor_sync(~0u, loss, off);
    if (lane == 0) sloss[warp] = loss;
  }
  if (EPI == EPI_STORE || EPI == EPI_OUT) return;
  __syncthreads();
  if (g.Ht)                            // 16 bytes a thread, along the rows
    for (int e = tid; e < BT * (BT / 8); e += GT_THREADS) {
      const int c = e / (BT / 8), r = e % (BT / 8) * 8;
      if (n0 + c < g.N)                // (rows up to the tile's end are allocated)
        *reinterpret_cast<uint4*>(g.Ht + (size_t)(n0 + c) * g.ldht + m0 + r) =
            *reinterpret_cast<const uint4*>(tr + c * TLD + r);
    }
  if (EPI == EPI_MSE && tid == 0)
    g.lpart[m0 / BT] = (sloss[0] + sloss[1]) + (sloss[2] + sloss[3]);
}

template <int BT, int BK, int EPI>
__global__ void __launch_bounds__(GT_THREADS) gemm_kernel(const __grid_constant__ GemmArgs g) {
  __shared__ __align__(16) __nv_bfloat16 sm[GT_STAGES][2][BT * (BK + 8)];
  __shared__ float sloss[4];
  after_previous();
  gemm_tile<BT, BK, EPI>(g, blockIdx.x, sm, sloss);
}

// dW and the bias gradients of all layers in one launch: the tiles of dW by layer,
// then the column sums.  Each of these blocks runs through all rows of the batch in
// order, so in a launch per layer (with dH) they were what it waited for: a step of
// 1024 rows 81 -> 69 us, of 4096 204 -> 122 (width 256, depth 4).
constexpr int ML_MAX = 16;                       // layers
struct GradArgs {
  int L, tiles[ML_MAX + 1], sums[ML_MAX + 1];
  GemmArgs w[ML_MAX];
  SumArgs s[ML_MAX];
};
__global__ void __launch_bounds__(GT_THREADS) grad_kernel(const __grid_constant__ GradArgs a) {
  __shared__ __align__(16) __nv_bfloat16 sm[GT_STAGES][2][GT_S * (GT_SK + 8)];
  __shared__ float sloss[4];
  static_assert(sizeof(sm) >= GT_STAGES * CS_ROWS * CS_COLS * 4, "stages of the sums");
  after_previous();
  const int b = blockIdx.x, b2 = b - a.tiles[a.L];
  int l = 0;
  if (b2 < 0) {
    while (b >= a.tiles[l + 1]) ++l;
    const GemmArgs g = a.w[l];
    gemm_tile<GT_S, GT_SK, EPI_STORE>(g, b - a.tiles[l], sm, sloss);
  } else {
    while (b2 >= a.sums[l + 1]) ++l;
    const SumArgs s = a.s[l];
    column_sums(s, b2 - a.sums[l], reinterpret_cast<float*>(&sm[0][0][0]));
  }
}

// one layer's view for the update: weights at w, bias behind them
struct LayerArgs {
  int dout, din, dout_pad, din_pad;
  int64_t off;                                   // into the flat parameters
  __nv_bfloat16 *Wb, *Wt;
};
struct UpdateArgs {
  LayerArgs l[ML_MAX];
};
struct LossArgs {                                // squares per row tile -> *loss
  int tiles;
  const float* part;
  float scale;
  float* loss;
};

// by one warp
__device__ void batch_loss(const LossArgs& u) {
  float s = 0.f;
  for (int t = threadIdx.x & 31; t < u.tiles; t += 32) s += u.part[t];
#pragma unroll
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(~0u, s, off);
  if (threadIdx.x == 0) *u.loss = s * u.scale;
}

// the loss without an update
__global__ void loss_kernel(LossArgs u) {
  after_previous();
  batch_loss(u);
}

// Adam and the new BF16 copies: blocks (32 x 32 tile of W, layer), W^T through
// shared memory; the block behind a layer's tiles takes its bias, and in layer 0
// the loss
__global__ void __launch_bounds__(256)
adam_kernel(UpdateArgs u, LossArgs ls, float* __restrict__ p, const float* __restrict__ g,
            float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2, float eps,
            float c1, float c2) {
  __shared__ __nv_bfloat16 tr[32][34];
  const LayerArgs& a = u.l[blockIdx.y];
  const int tx = (a.din + 31) / 32, nt = tx * ((a.dout + 31) / 32), t = blockIdx.x;
  if (t > nt) return;
  after_previous();
  auto step = [&](int64_t i, float gi) {
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    return p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  };
  if (t == nt) {
    for (int c = threadIdx.x; c < a.dout; c += blockDim.x) {
      const int64_t i = a.off + (int64_t)a.dout * a.din + c;
      step(i, g[i]);
    }
    if (blockIdx.y == 0 && threadIdx.x < 32) batch_loss(ls);
    return;
  }
  const int r0 = t / tx * 32, c0 = t % tx * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 32; q += 8) {
    const int r = r0 + y + q, c = c0 + x;
    if (r < a.dout && c < a.din) {
      const int64_t i = a.off + (int64_t)r * a.din + c;
      const __nv_bfloat16 b = __float2bfloat16(step(i, g[i]));
      a.Wb[(size_t)r * a.din_pad + c] = b;
      tr[y + q][x] = b;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 32; q += 8) {
    const int r = r0 + x, c = c0 + y + q;
    if (r < a.dout && c < a.din) a.Wt[(size_t)c * a.dout_pad + r] = tr[x][y + q];
  }
}

// fp32 weights [rows][cols] -> bf16 W [rows_pad][cols_pad] and W^T [cols_pad][rows_pad]
__global__ void pack_weights_kernel(int rows, int cols, int rows_pad, int cols_pad,
                                    const float* __restrict__ w, __nv_bfloat16* __restrict__ Wb,
                                    __nv_bfloat16* __restrict__ Wt) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < rows_pad * cols_pad;
       e += gridDim.x * blockDim.x) {
    const int r = e / cols_pad, c = e % cols_pad;
    const float x = (r < rows && c < cols) ? w[(size_t)r * cols + c] : 0.f;
    const __nv_bfloat16 b = __float2bfloat16(x);
    Wb[e] = b;
    Wt[(size_t)c * rows_pad + r] = b;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
struct kls_mlp {
  int device = 0, width = 256, depth = 4, cap = 0;  // depth = number of linear layers
  std::vector<int> din, dout, din_pad, dout_pad;    // per layer
  std::vector<int64_t> woff, boff;                  // offsets into the flat fp32 params
  int64_t nparams = 0;
  void* pslab = nullptr;                            // the allocation of p .. Wt
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  std::vector<__nv_bfloat16*> Wb, Wt;
  // activations for a batch of `cap` rows, of a training pass for `tcap`
  int tcap = 0;
  void *hslab = nullptr, *tslab = nullptr, *rslab = nullptr;   // their allocations, and X .. idx
  std::vector<float*> Z;                             // pre-activations [cap][dout_pad]
  std::vector<__nv_bfloat16*> H, Ht;                 // H[l]: input of layer l [cap][din_pad]
  __nv_bfloat16 *dZ[2] = {nullptr, nullptr};         // bf16 [cap][width], by turns
  std::vector<__nv_bfloat16*> dZt;                   // bf16 [dout_pad][cap] of every layer
  std::vector<float*> dZf;                           // fp32 [cap][dout_pad]
  bool lean = false;                                 // dZt and dZf of one layer only, by turns
  int ltiles = 0;                                    // row tiles of the last batch
  float* lpart = nullptr;                            // squared errors per row tile
  int rows = 0, steps = 0;                           // capacity of the buffers below
  float *Xd = nullptr, *Td = nullptr, *Yd = nullptr; // rows of a call
  int* idx = nullptr;                                // [rows] shuffled order
  float* loss = nullptr;                             // [steps] of an epoch
  int64_t step = 0;
  cudaStream_t stream = nullptr;
  std::string err;
};

namespace {

int mfail(kls_mlp* m, const std::string& s) {
  if (m) m->err = s;
  return kls_fail(nullptr, KLS_ERR_CUDA, s);
}
#define ML_CK(m, call)                                                            \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) {                                                      \
      cudaGetLastError();    /* reported here */                                  \
      return mfail(m, std::string(#call) + ": " + cudaGetErrorString(e_));        \
    }                                                                             \
  } while (0)

// activations of n rows; `train`: and all that a training pass leaves
int ensure_cap(kls_mlp* m, int n, bool train) {
  const int L = m->depth, cap = ((n + 63) / 64) * 64;
  if (n > m->cap) {
    m->cap = 0;
    cudaFree(m->hslab);
    KlsSlab b;
    m->H.assign(L, nullptr);           // inputs of the layers 1 .. L - 1
    for (int l = 1; l < L; ++l) b.add(&m->H[l], (size_t)cap * m->din_pad[l]);
    ML_CK(m, b.alloc(&m->hslab));
    m->cap = cap;
  }
  if (train && n > m->tcap) {
    m->tcap = 0;
    cudaFree(m->tslab);
    m->Z.assign(L, nullptr);           // layers 0 .. L - 2
    m->Ht.assign(L, nullptr);          // inputs of all layers
    m->dZt.assign(L, nullptr);
    m->dZf.assign(L, nullptr);
    // dZt and dZf of every layer let one launch take all of dW; where they do not fit
    // (14 against 8 bytes a row and hidden unit), those of one layer
    cudaError_t e = cudaSuccess;
    for (int lean = 0; lean < 2; ++lean) {
      KlsSlab b;
      m->lean = lean;
      for (int l = 0; l < L; ++l) {
        const size_t in = (size_t)cap * m->din_pad[l], out = (size_t)cap * m->dout_pad[l];
        if (l < L - 1) b.add(&m->Z[l], out);
        b.add(&m->Ht[l], in);
        if (!lean) b.add(&m->dZt[l], out).add(&m->dZf[l], out);
      }
      if (lean) b.add(&m->dZt[0], (size_t)cap * m->width).add(&m->dZf[0], (size_t)cap * m->width);
      for (int q = 0; q < 2; ++q) b.add(&m->dZ[q], (size_t)cap * m->width);
      b.add(&m->lpart, (size_t)cap / GT_S);
      e = b.alloc(&m->tslab);
      if (e != cudaErrorMemoryAllocation) break;
    }
    ML_CK(m, e);
    for (int l = 1; m->lean && l < L; ++l) { m->dZt[l] = m->dZt[0]; m->dZf[l] = m->dZf[0]; }
    m->tcap = cap;
  }
  return KLS_OK;
}

// X, T, Y and the order of n rows; losses of `steps` steps
int ensure_rows(kls_mlp* m, int n, int steps) {
  if (n > m->rows) {
    m->rows = 0;
    cudaFree(m->rslab);
    KlsSlab b;
    b.add(&m->Xd, (size_t)n * ML_IN).add(&m->Td, (size_t)n * ML_OUT);
    b.add(&m->Yd, (size_t)n * ML_OUT).add(&m->idx, n);
    ML_CK(m, b.alloc(&m->rslab));
    m->rows = n;
  }
  if (steps > m->steps) {
    m->steps = 0;
    cudaFree(m->loss);
    m->loss = nullptr;
    ML_CK(m, cudaMalloc(&m->loss, (size_t)steps * 4));
    m->steps = steps;
  }
  return KLS_OK;
}

template <typename... P, typename... A>
int launch(kls_mlp* m, void (*kernel)(P...), dim3 grid, int threads, A... args) {
  cudaLaunchConfig_t c = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.stream = m->stream;
  c.attrs = at;
  c.numAttrs = 1;
  ML_CK(m, cudaLaunchKernelEx(&c, kernel, P(args)...));
  return KLS_OK;
}

int tiles(const GemmArgs& g, int t) { return ((g.N + t - 1) / t) * ((g.M + t - 1) / t); }

// The large tile from two of its blocks per SM on: there it reads half as much of
// the operands per product (forward of 32768 rows, width 256, depth 4, host to host:
// 189 against 222 us); below that the small one has the more SMs at work (a
// training step of 1024 rows is a quarter slower in large ones; 8192 rows are alike,
// 85 us).
template <int EPI>
int gemm(kls_mlp* m, const GemmArgs& g) {
  const bool large = tiles(g, GT_L) >= 296;
  const int t = large ? GT_L : GT_S;
  if (EPI == EPI_MSE) m->ltiles = (g.M + t - 1) / t;
  return launch(m, large ? gemm_kernel<GT_L, GT_LK, EPI> : gemm_kernel<GT_S, GT_SK, EPI>,
                dim3(tiles(g, t)), GT_THREADS, g);
}

int pack_all(kls_mlp* m) {
  for (int l = 0; l < m->depth; ++l) {
    int n = m->dout_pad[l] * m->din_pad[l];
    pack_weights_kernel<<<(n + 255) / 256, 256, 0, m->stream>>>(
        m->dout[l], m->din[l], m->dout_pad[l], m->din_pad[l], m->p + m->woff[l], m->Wb[l], m->Wt[l]);
    ML_CK(m, cudaGetLastError());
  }
  return KLS_OK;
}

// forward over n rows of X (rows idx, or in order from row0 on); train: keeps Z and the
// transposes, and ends in the gradient of the loss; else the outputs to m->Yd
int forward(kls_mlp* m, int n, const int* idx, int row0, bool train) {
  const int L = m->depth;
  for (int l = 0; l < L; ++l) {
    GemmArgs g{};
    g.M = n; g.N = m->dout_pad[l]; g.K = m->din_pad[l];
    g.A = m->H[l]; g.lda = m->din_pad[l];
    g.B = m->Wb[l]; g.ldb = m->din_pad[l];
    // (the last layer's bias covers 3 outputs; the padded ones read zeros behind it)
    g.bias = m->p + m->boff[l];
    g.ldht = m->tcap;
    g.idx = idx;
    if (l == 0) {
      g.X = m->Xd + (size_t)row0 * ML_IN;
      g.Xt = train ? m->Ht[0] : nullptr;
    }
    int r;
    if (l < L - 1) {
      g.H = m->H[l + 1]; g.ldh = m->din_pad[l + 1];
      if (train) {
        g.C = m->Z[l]; g.ldc = m->dout_pad[l];
        g.Ht = m->Ht[l + 1];
      }
      r = gemm<EPI_GELU>(m, g);
    } else if (train) {
      g.T = m->Td + (size_t)row0 * ML_OUT;
      g.C = m->dZf[l]; g.ldc = m->dout_pad[l];
      g.H = m->dZ[0]; g.ldh = m->dout_pad[l];
      g.Ht = m->dZt[l];
      g.lpart = m->lpart;
      r = gemm<EPI_MSE>(m, g);
    } else {
      g.C = m->Yd;
      r = gemm<EPI_OUT>(m, g);
    }
    if (r) return r;
  }
  return KLS_OK;
}

// backward from the gradient that a training forward leaves in dZ[0]
int backward(kls_mlp* m, int n) {
  const int L = m->depth;
  GradArgs a{};
  // dW and bias gradients of the layers collected in a
  auto grads = [&]() {
    for (int i = 0; i < a.L; ++i) {
      a.tiles[i + 1] = a.tiles[i] + tiles(a.w[i], GT_S);
      a.sums[i + 1] = a.sums[i] + (a.s[i].N + CS_COLS - 1) / CS_COLS;
    }
    return launch(m, grad_kernel, dim3(a.tiles[a.L] + a.sums[a.L]), GT_THREADS, a);
  };
  for (int l = L - 1, q = 0; l >= 0; --l, q ^= 1) {
    // dW_l [dout][din] = dZ_l^T (dout x n) * H_l (n x din): A = dZt_l [dout_pad][cap], B = Ht_l
    GemmArgs& w = a.w[a.L];
    w.M = m->dout[l]; w.N = m->din[l]; w.K = n;
    w.A = m->dZt[l]; w.lda = m->tcap;
    w.B = m->Ht[l]; w.ldb = m->tcap;
    w.C = m->g + m->woff[l]; w.ldc = m->din[l];
    a.s[a.L++] = {n, m->dout[l], m->dout_pad[l], m->dZf[l], m->g + m->boff[l]};
    int r;
    if (m->lean) {                     // before the next layer takes their place
      if ((r = grads())) return r;
      a.L = 0;
    }
    if (l == 0) break;
    // dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1}): A = dZ [n][dout_pad], B = Wt_l [din_pad][dout_pad]
    GemmArgs h{};
    h.M = n; h.N = m->din_pad[l]; h.K = m->dout_pad[l];
    h.A = m->dZ[q]; h.lda = m->dout_pad[l];
    h.B = m->Wt[l]; h.ldb = m->dout_pad[l];
    h.Zin = m->Z[l - 1]; h.ldz = m->dout_pad[l - 1];
    h.C = m->dZf[l - 1]; h.ldc = m->din_pad[l];
    h.H = m->dZ[q ^ 1]; h.ldh = m->din_pad[l];
    h.Ht = m->dZt[l - 1]; h.ldht = m->tcap;
    if ((r = gemm<EPI_GELU_BWD>(m, h))) return r;
  }
  return m->lean ? KLS_OK : grads();
}

LossArgs loss_args(const kls_mlp* m, int n, float* loss) {
  return {m->ltiles, m->lpart, 1.f / (float)(n * ML_OUT), loss};
}

// gradients into m->g and the loss by row tiles
int grad_batch(kls_mlp* m, int n, const int* idx, int row0) {
  int r = forward(m, n, idx, row0, true);
  return r ? r : backward(m, n);
}

}  // namespace

extern "C" {

int kls_mlp_create(int device, int width, int depth, uint64_t seed, kls_mlp** out) {
  if (!out || width < 16 || width % 16 || depth < 2 || depth > 16)
    return kls_fail(nullptr, KLS_ERR_CONFIG, "kls_mlp_create: bad arguments");
  *out = nullptr;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return kls_fail(nullptr, KLS_ERR_CUDA, cudaGetErrorString(e));
  kls_mlp* m = new kls_mlp();
  m->device = device; m->width = width; m->depth = depth;
  for (int l = 0; l < depth; ++l) {
    int di = l == 0 ? ML_IN : width, dO = l == depth - 1 ? ML_OUT : width;
    m->din.push_back(di); m->dout.push_back(dO);
    m->din_pad.push_back(l == 0 ? ML_PAD : width);
    m->dout_pad.push_back(l == depth - 1 ? ML_PAD : width);
    m->woff.push_back(m->nparams); m->nparams += (int64_t)di * dO;
    m->boff.push_back(m->nparams); m->nparams += dO;
  }
  // the last bias is read for all 16 padded outputs: reserve 13 zero floats after it
  const int64_t alloc = m->nparams + ML_PAD;
  std::vector<float> h(alloc, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < depth; ++l) {
    const float bound = 1.0f / std::sqrt((float)m->din[l]);   // uniform(-1/sqrt(fan_in), ..)
    std::uniform_real_distribution<float> U(-bound, bound);
    for (int64_t i = 0; i < (int64_t)m->din[l] * m->dout[l]; ++i) h[m->woff[l] + i] = U(rng);
    for (int i = 0; i < m->dout[l]; ++i) h[m->boff[l] + i] = U(rng);
  }
  KlsSlab b;
  b.add(&m->p, alloc).add(&m->g, alloc).add(&m->m, alloc).add(&m->v, alloc);
  m->Wb.assign(depth, nullptr);
  m->Wt.assign(depth, nullptr);
  for (int l = 0; l < depth; ++l) {
    const size_t n = (size_t)m->dout_pad[l] * m->din_pad[l];
    b.add(&m->Wb[l], n).add(&m->Wt[l], n);
  }
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
      b.alloc(&m->pslab) != cudaSuccess) {
    kls_mlp_destroy(m);
    return kls_fail(nullptr, KLS_ERR_OOM, "kls_mlp_create: device allocation failed");
  }
  cudaMemcpyAsync(m->p, h.data(), alloc * 4, cudaMemcpyHostToDevice, m->stream);
  cudaMemsetAsync(m->g, 0, alloc * 4, m->stream);
  cudaMemsetAsync(m->m, 0, alloc * 4, m->stream);
  cudaMemsetAsync(m->v, 0, alloc * 4, m->stream);
  int r = pack_all(m);
  if (!r && cudaStreamSynchronize(m->stream) != cudaSuccess)
    r = kls_fail(nullptr, KLS_ERR_CUDA, "kls_mlp_create: init failed");
  if (r) {
    kls_mlp_destroy(m);
    return r;
  }
  *out = m;
  return KLS_OK;
}

int kls_mlp_destroy(kls_mlp* m) {
  if (!m) return KLS_OK;
  cudaSetDevice(m->device);
  if (m->stream) cudaStreamSynchronize(m->stream);
  for (void* x : {m->pslab, m->hslab, m->tslab, m->rslab, (void*)m->loss}) cudaFree(x);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
  return KLS_OK;
}

int kls_mlp_num_params(const kls_mlp* m, int64_t* n) {
  if (!m || !n) return KLS_ERR_CONFIG;
  *n = m->nparams;
  return KLS_OK;
}

int kls_mlp_get_params(kls_mlp* m, float* params) {
  if (!m || !params) return KLS_ERR_CONFIG;
  cudaSetDevice(m->device);
  ML_CK(m, cudaMemcpy(params, m->p, m->nparams * 4, cudaMemcpyDeviceToHost));
  return KLS_OK;
}

int kls_mlp_set_params(kls_mlp* m, const float* params) {
  if (!m || !params) return KLS_ERR_CONFIG;
  cudaSetDevice(m->device);
  ML_CK(m, cudaMemcpyAsync(m->p, params, m->nparams * 4, cudaMemcpyHostToDevice, m->stream));
  int r = pack_all(m);
  if (r) return r;
  ML_CK(m, cudaStreamSynchronize(m->stream));
  return KLS_OK;
}

// Inference: X [n][5] host -> Y [n][3] host
int kls_mlp_forward(kls_mlp* m, const float* X, int n, float* Y) {
  if (!m || n < 0 || (n && (!X || !Y))) return KLS_ERR_CONFIG;
  cudaSetDevice(m->device);
  const int chunk = 1 << 16;
  for (int s = 0; s < n; s += chunk) {
    int nb = std::min(chunk, n - s);
    int r = ensure_cap(m, nb, false);
    if (r || (r = ensure_rows(m, nb, 0))) return r;
    ML_CK(m, cudaMemcpyAsync(m->Xd, X + (size_t)s * ML_IN, (size_t)nb * ML_IN * 4,
                             cudaMemcpyHostToDevice, m->stream));
    if ((r = forward(m, nb, nullptr, 0, false))) return r;
    ML_CK(m, cudaMemcpyAsync(Y + (size_t)s * ML_OUT, m->Yd, (size_t)nb * ML_OUT * 4,
                             cudaMemcpyDeviceToHost, m->stream));
    ML_CK(m, cudaStreamSynchronize(m->stream));
  }
  return KLS_OK;
}

// Loss and full-batch gradients (no update), for gradient checks
int kls_mlp_grad(kls_mlp* m, const float* X, const float* T, int n, float* grads, float* loss) {
  if (!m || n < 1 || !X || !T) return KLS_ERR_CONFIG;
  cudaSetDevice(m->device);
  int r = ensure_cap(m, n, true);
  if (r || (r = ensure_rows(m, n, 1))) return r;
  ML_CK(m, cudaMemcpyAsync(m->Xd, X, (size_t)n * ML_IN * 4, cudaMemcpyHostToDevice, m->stream));
  ML_CK(m, cudaMemcpyAsync(m->Td, T, (size_t)n * ML_OUT * 4, cudaMemcpyHostToDevice, m->stream));
  if ((r = grad_batch(m, n, nullptr, 0))) return r;
  if ((r = launch(m, loss_kernel, dim3(1), 32, loss_args(m, n, m->loss)))) return r;
  if (grads) ML_CK(m, cudaMemcpyAsync(grads, m->g, m->nparams * 4, cudaMemcpyDeviceToHost, m->stream));
  if (loss) ML_CK(m, cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->stream));
  ML_CK(m, cudaStreamSynchronize(m->stream));
  return KLS_OK;
}

// Adam training: epochs over shuffled minibatches; loss_hist[e] = mean batch loss
int kls_mlp_train(kls_mlp* m, const float* X, const float* T, int n, int epochs, int batch,
                  float lr, uint64_t seed, float* loss_hist) {
  if (!m || n < 1 || batch < 1 || epochs < 0 || !X || !T) return KLS_ERR_CONFIG;
  if (epochs == 0) return KLS_OK;      // (X and T are the caller's again: no copy of them)
  cudaSetDevice(m->device);
  batch = std::min(batch, n);
  const int steps = n / batch;
  // up to ML_ROWS rows are on the device for the whole call and gathered there; of
  // more, a segment of batches at a time in the epoch's order
  const bool all = n <= ML_ROWS;
  const int seg = all ? n : std::max(1, ML_ROWS / batch) * batch;
  int r = ensure_cap(m, batch, true);
  if (r || (r = ensure_rows(m, seg, steps))) return r;
  int tiles_w = 1;                                       // blocks of the update, per layer
  for (int l = 0; l < m->depth; ++l)
    tiles_w = std::max(tiles_w, ((m->din[l] + 31) / 32) * ((m->dout[l] + 31) / 32) + 1);
  auto upload = [&](const float* x, const float* t, int rows) -> int {
    ML_CK(m, cudaMemcpyAsync(m->Xd, x, (size_t)rows * ML_IN * 4, cudaMemcpyHostToDevice, m->stream));
    ML_CK(m, cudaMemcpyAsync(m->Td, t, (size_t)rows * ML_OUT * 4, cudaMemcpyHostToDevice, m->stream));
    return KLS_OK;
  };
  std::vector<float> xb, tb;
  if (all && (r = upload(X, T, n))) return r;
  UpdateArgs u{};
  for (int l = 0; l < m->depth; ++l)
    u.l[l] = {m->dout[l], m->din[l], m->dout_pad[l], m->din_pad[l], m->woff[l], m->Wb[l], m->Wt[l]};
  std::vector<int> idx(n);
  for (int i = 0; i < n; ++i) idx[i] = i;
  std::mt19937_64 rng(seed);
  std::vector<float> ls(steps);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::shuffle(idx.begin(), idx.end(), rng);
  for (int ep = 0; ep < epochs; ++ep) {
    if (all)
      ML_CK(m, cudaMemcpyAsync(m->idx, idx.data(), (size_t)n * 4, cudaMemcpyHostToDevice,
                               m->stream));
    for (int s = 0; s < steps; ++s) {
      const int64_t first = (int64_t)s * batch;
      if (!all && first % seg == 0) {
        const int rows = (int)std::min<int64_t>(seg, (int64_t)steps * batch - first);
        ML_CK(m, cudaStreamSynchronize(m->stream));      // the rows before are used and copied
        xb.resize((size_t)rows * ML_IN);
        tb.resize((size_t)rows * ML_OUT);
        for (int i = 0; i < rows; ++i) {
          const size_t q = idx[first + i];
          std::copy_n(X + q * ML_IN, ML_IN, xb.begin() + (size_t)i * ML_IN);
          std::copy_n(T + q * ML_OUT, ML_OUT, tb.begin() + (size_t)i * ML_OUT);
        }
        if ((r = upload(xb.data(), tb.data(), rows))) return r;
      }
      if ((r = grad_batch(m, batch, all ? m->idx + first : nullptr, all ? 0 : (int)(first % seg))))
        return r;
      ++m->step;
      const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
      if ((r = launch(m, adam_kernel, dim3(tiles_w, m->depth), 256,
                      u, loss_args(m, batch, m->loss + s), m->p, m->g, m->m, m->v, lr, b1, b2, eps,
                      c1, c2)))
        return r;
    }
    if (ep + 1 < epochs) std::shuffle(idx.begin(), idx.end(), rng);
    ML_CK(m, cudaMemcpyAsync(ls.data(), m->loss, (size_t)steps * 4, cudaMemcpyDeviceToHost,
                             m->stream));
    ML_CK(m, cudaStreamSynchronize(m->stream));
    double lsum = 0.0;
    for (float l : ls) lsum += l;
    if (loss_hist) loss_hist[ep] = steps ? (float)(lsum / steps) : 0.f;
  }
  return KLS_OK;
}

}  // extern "C"
