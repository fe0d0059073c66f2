/*
 * Learned density of states: a small MLP (BF16 weights and activations,
 * FP32 accumulation and master weights) that maps KPM moments estimated from
 * a few random vectors to the moments of many vectors.  Training and
 * inference run on this file's kernels:
 *
 *   k_gemm_bf16   C = op(A) op(B) on the tensor cores (warp-level
 *                 mma.sync m16n8k16, BF16 inputs, FP32 accumulators), 32x32
 *                 tiles, operands staged in shared memory (either operand
 *                 may be transposed), with fused epilogues:
 *                 bias + GELU (forward), bias (output layer), GELU'
 *                 (backward through an activation), plain store (weight
 *                 gradients, with the bias gradients' column sums);
 *   k_mse         dY = 2 (Y - T) / (B * nout) on the real outputs, and the
 *                 loss (deterministic block-ordered sum);
 *   k_adam        Adam on the FP32 master weights, then the BF16 copies.
 *
 * Layer l maps K_l inputs to N_l outputs (dimensions padded to multiples of
 * 16 with zero weights); activations are row-major [batch][features].
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "gpu.cuh"
#include "gpu_device.cuh"

namespace pv {

typedef __nv_bfloat16 bf16;

constexpr int kGT = 32;    /* block tile (M and N) */
constexpr int kGKC = 320;  /* k staged at once (a multiple of 16) */

enum { EPI_STORE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_DGELU = 3 };

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

__device__ __forceinline__ void mma_bf16_16816(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

/* 16 bytes to shared memory, zeros when !ok */
__device__ __forceinline__ void cp16(void *dst, const void *src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}

__device__ __forceinline__ void ldm4(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldm4t(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

/* db[n] = sum_m dZ[m][n], rows in order, for the 32 columns from n0 on: the
 * block's warps stage 64 rows at a time and warp 0 adds them */
__device__ __forceinline__ void colsum(int Bn, int N, int n0, const float *dZ, int ld,
                                       float *__restrict__ db, float *sh) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, n = n0 + lane;
  float s = 0.f, next[16];
  auto fetch = [&](int t) {
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const int m = t + wib * 16 + q;
      next[q] = m < Bn && n < N ? dZ[(size_t)m * ld + n] : 0.f;
    }
  };
  fetch(0);
  for (int t = 0, buf = 0; t < Bn; t += 64, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < 16; q++) sh[(buf * 64 + wib * 16 + q) * 32 + lane] = next[q];
    __syncthreads();
    fetch(t + 64);
    if (wib == 0) {
      const int m = Bn - t < 64 ? Bn - t : 64;
#pragma unroll 16
      for (int r = 0; r < m; r++) s += sh[(buf * 64 + r) * 32 + lane];
    }
  }
  if (wib == 0 && n < N) db[n] = s;
}

/* C[m][n] = sum_k A'(m,k) B'(k,n) for m < M, n < N, with
 * A'(m,k) = TA ? A[k*lda + m] : A[m*lda + k] and
 * B'(k,n) = TB ? B[n*ldb + k] : B[k*ldb + n]; out-of-range elements are 0.
 * Every extent along a row of A or B is a multiple of 16 (padded layer
 * sizes), so rows are staged in 16-byte copies; the batch, which is not,
 * runs along the rows' index.  128 threads: warp w owns the 16 x 16 piece
 * (w / 2, w % 2) of a 32 x 32 tile.  Epilogue (row m, column n):
 *   EPI_STORE      C = acc; one more block per row of tiles forms the column
 *                  sums db of the FP32 dZ (zp, the K rows of C's m columns)
 *   EPI_BIAS       C = acc + bias[n]
 *   EPI_BIAS_GELU  C = z = acc + bias[n];  act = bf16(gelu(z))
 *   EPI_DGELU      C = g = acc * gelu'(zp[m][n]);  act = bf16(g)
 * What bounds it is latency: a layer of 128 x 256 x 304 is 20 MFLOP on a few
 * dozen blocks.  So all of K (up to kGKC) is staged at once, in one round
 * trip, and the k steps run without a barrier: a forward layer 26.7 -> 5.5 us
 * against 64 x 64 tiles staged 16 deep element by element (ten blocks, a
 * round trip per k step).  The k steps come in the same order: the same bits. */
template <bool TA, bool TB, int EPI>
__global__ void __launch_bounds__(128)
    k_gemm_bf16(int M, int N, int K, const bf16 *A, int lda,
                const bf16 *__restrict__ B, int ldb, float *__restrict__ C, int ldc,
                const float *__restrict__ bias, bf16 *__restrict__ act, int ldact,
                const float *zp, int ldzp, float *__restrict__ db) {
  /* a tile's rows: k along them (32 rows of kGKC + 8) or across (kGKC rows of
   * 32 + 8); the padding makes the eight rows of an ldmatrix hit eight banks */
  constexpr int LDK = kGKC + 8, LDT = kGT + 8;
  constexpr int SZ = kGT * LDK > kGKC * LDT ? kGT * LDK : kGKC * LDT;
  extern __shared__ __align__(16) bf16 gsm[];
  bf16 *As = gsm, *Bs = gsm + SZ;
  /* the rows, which are the batch in a forward layer, along x: y ends at 65535 */
  if (EPI == EPI_STORE && (int)blockIdx.y * kGT >= N) {
    pdl_wait_then_release();
    colsum(K, M, (int)blockIdx.x * kGT, zp, ldzp, db, (float *)gsm);
    return;
  }
  const int m0 = blockIdx.x * kGT, n0 = blockIdx.y * kGT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
  float acc[2][4], pre[2][4] = {}; /* pre: what the epilogue multiplies by */
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) acc[j][q] = 0.f;
  for (int k0 = 0; k0 < K; k0 += kGKC) {
    const int kc = K - k0 < kGKC ? K - k0 : kGKC, kr = (kc + 15) / 16 * 16;
    if (k0) __syncthreads();
    auto stage = [&](bf16 *S, const bf16 *G, int ld, bool across, int o, int lim) {
      if (across) { /* row = k, 32 elements from column o on */
        for (int t = threadIdx.x; t < kr * (kGT / 8); t += 128) {
          const int r = t / (kGT / 8), c = t % (kGT / 8) * 8;
          const bool ok = r < kc && o + c < lim;
          cp16(S + r * LDT + c, ok ? G + (size_t)(k0 + r) * ld + o + c : G, ok);
        }
      } else { /* row = m or n, kr elements from k0 on */
        const int per = kr / 8;
        for (int t = threadIdx.x; t < kGT * per; t += 128) {
          const int r = t / per, c = t % per * 8;
          const bool ok = o + r < lim && c < kc;
          cp16(S + r * LDK + c, ok ? G + (size_t)(o + r) * ld + k0 + c : G, ok);
        }
      }
    };
    /* B (weights, or a layer's stored input) is never what the launch before
     * this one wrote, A may be */
    stage(Bs, B, ldb, !TB, n0, N);
    if (k0 == 0) {
      pdl_wait_then_release();
      if (EPI == EPI_DGELU) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int m = m0 + wm + gid + (q >= 2 ? 8 : 0), n = n0 + wn + 8 * j + 2 * tig + (q & 1);
            pre[j][q] = m < M && n < N ? zp[(size_t)m * ldzp + n] : 0.f;
          }
      }
    }
    stage(As, A, lda, TA, m0, M);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    /* matrix q of an ldmatrix.x4 is addressed by lanes 8 q .. 8 q + 7.  A: rows
     * +0, +8, +0, +8 at k +0, +0, +8, +8.  B: columns +0, +0, +8, +8 at k +0,
     * +8, +0, +8 (two 8-column tiles). */
    const int q = lane >> 3, r8 = lane & 7;
    const int am = wm + (q & 1) * 8, ak = (q >> 1) * 8, bn = wn + (q >> 1) * 8, bk = (q & 1) * 8;
    for (int kk = 0; kk < kr; kk += 16) {
      uint32_t af[4], bf[4];
      if constexpr (TA)
        ldm4t(af, smem_addr(As + (kk + ak + r8) * LDT + am));
      else
        ldm4(af, smem_addr(As + (am + r8) * LDK + kk + ak));
      if constexpr (TB)
        ldm4(bf, smem_addr(Bs + (bn + r8) * LDK + kk + bk));
      else
        ldm4t(bf, smem_addr(Bs + (kk + bk + r8) * LDT + bn));
      mma_bf16_16816(acc[0], af, bf);
      mma_bf16_16816(acc[1], af, bf + 2);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int m = m0 + wm + gid + (q >= 2 ? 8 : 0);
      const int n = n0 + wn + 8 * j + 2 * tig + (q & 1);
      if (m >= M || n >= N) continue;
      float v = acc[j][q];
      if (EPI == EPI_BIAS || EPI == EPI_BIAS_GELU) v += bias[n];
      if (EPI == EPI_DGELU) v *= gelu_grad(pre[j][q]);
      C[(size_t)m * ldc + n] = v;
      if (EPI == EPI_BIAS_GELU) act[(size_t)m * ldact + n] = __float2bfloat16(gelu(v));
      if (EPI == EPI_DGELU) act[(size_t)m * ldact + n] = __float2bfloat16(v);
    }
}

/* dY = 2 (Y - T) / (B * nout) on columns < nout (0 elsewhere), bf16 copy,
 * and the mean squared error: per-block sums, the last block adds them in
 * block order */
__global__ void k_mse(int Bn, int ld, int nout, const float *Y,
                      const float *__restrict__ T, int ldt, float *__restrict__ dY,
                      bf16 *__restrict__ dYh, double *partials, unsigned *counter, float *loss) {
  __shared__ double sh[256];
  __shared__ bool am_last;
  pdl_wait_then_release();
  const double scale = 2.0 / ((double)Bn * nout);
  double s = 0.0;
  const long tot = (long)Bn * ld;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < tot; i += (long)gridDim.x * blockDim.x) {
    const int m = (int)(i / ld), n = (int)(i % ld);
    float g = 0.f;
    if (n < nout) {
      const float d = Y[i] - T[(size_t)m * ldt + n];
      s += (double)d * d;
      g = (float)(scale * d);
    }
    dY[i] = g;
    dYh[i] = __float2bfloat16(g);
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = sh[0];
    __threadfence();
    am_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (am_last && threadIdx.x == 0) {
    __threadfence();
    double t = 0.0;
    for (unsigned b = 0; b < gridDim.x; b++) t += __ldcg(partials + b);
    *loss = (float)(t / ((double)Bn * nout));
    *counter = 0;
  }
}

/* Adam (Kingma & Ba, 2015) with bias correction on FP32 master weights;
 * entries with mask 0 (padding) stay 0 */
__global__ void k_adam(long np, float *__restrict__ p, const float *g,
                       float *__restrict__ m1, float *__restrict__ m2, const uint8_t *__restrict__ mask,
                       bf16 *__restrict__ ph, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  pdl_wait_then_release();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < np; i += (long)gridDim.x * blockDim.x) {
    if (!mask[i]) {
      p[i] = 0.f;
      ph[i] = __float2bfloat16(0.f);
      continue;
    }
    const float gi = g[i];
    const float a = b1 * m1[i] + (1.f - b1) * gi;
    const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float v = p[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[i] = v;
    ph[i] = __float2bfloat16(v);
  }
}

__global__ void k_to_bf16(long n, const float *__restrict__ x, bf16 *__restrict__ y) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

/* X [B][ld] (bf16, zero padding) from a row-major FP32 block [B][nin] */
__global__ void k_pack_input(int Bn, int nin, int ld, const float *x, bf16 *__restrict__ xh) {
  pdl_wait_then_release();
  const long tot = (long)Bn * ld;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < tot; i += (long)gridDim.x * blockDim.x) {
    const int m = (int)(i / ld), n = (int)(i % ld);
    xh[i] = __float2bfloat16(n < nin ? x[(size_t)m * nin + n] : 0.f);
  }
}

template <bool TA, bool TB, int EPI>
static int gemm(int M, int N, int K, const bf16 *A, int lda, const bf16 *B, int ldb, float *C, int ldc,
                const float *bias, bf16 *act, int ldact, const float *zp, int ldzp,
                float *db = nullptr) {
  if (M <= 0 || N <= 0) return 0;
  dim3 g((unsigned)((M + kGT - 1) / kGT), (unsigned)((N + kGT - 1) / kGT + (EPI == EPI_STORE)));
  /* two operands of at most kGKC x (kGT + 8) or kGT x (kGKC + 8) elements */
  constexpr size_t sm = 2 * sizeof(bf16) * (kGT * (kGKC + 8) > kGKC * (kGT + 8) ? kGT * (kGKC + 8) : kGKC * (kGT + 8));
  static_assert(sm >= 2 * 64 * 32 * sizeof(float), "the column sums stage two tiles");
  static const cudaError_t attr = cudaFuncSetAttribute(
      k_gemm_bf16<TA, TB, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (fail(attr, "cudaFuncSetAttribute")) return PEVSL_ERR_CUDA;
  launch_pdl_block(k_gemm_bf16<TA, TB, EPI>, g, 128, sm, ctx().stream, M, N, K, A, lda, B, ldb, C, ldc,
                   bias, act, ldact, zp, ldzp, db);
  return launched("gemm_bf16");
}

}  // namespace pv

using namespace pv;

/* ---------------------------------------------------------------- network */
struct pevsl_mlp {
  int nin, nout, width, layers; /* layers = number of linear maps */
  int kdim[8], ndim[8];         /* padded: K (inputs) and N (outputs) per layer */
  long woff[8], boff[8];        /* offsets of W_l (N x K, row-major) and b_l in the parameter block */
  long np;                      /* parameters incl. padding */
  float *p, *g, *m1, *m2;       /* device FP32: master, gradient, Adam moments */
  bf16 *ph;                     /* device BF16 copy of p */
  uint8_t *mask;                /* 1 for real parameters, 0 for padding */
  long step;
  int cap;                      /* batch capacity of the buffers */
  float *z[8];                  /* pre-activations [cap][N_l] */
  bf16 *a[9];                   /* a[0] = input, a[l+1] = gelu(z[l]) [cap][N_l] */
  float *dz;                    /* gradient of a pre-activation [cap][maxdim] (fp32) */
  bf16 *dzh[2];                 /* bf16 copies, ping-pong */
  float *loss;                  /* device scalar */
  double *partials;
  unsigned *counter;
};

static int pad16(int x) { return (x + 15) / 16 * 16; }

static void mlp_free_buffers(pevsl_mlp *net) {
  for (int l = 0; l < 8; l++) {
    cudaFree(net->z[l]);
    net->z[l] = nullptr;
  }
  for (int l = 0; l < 9; l++) {
    cudaFree(net->a[l]);
    net->a[l] = nullptr;
  }
  cudaFree(net->dz);
  cudaFree(net->dzh[0]);
  cudaFree(net->dzh[1]);
  net->dz = nullptr;
  net->dzh[0] = net->dzh[1] = nullptr;
  net->cap = 0;
}

static int mlp_reserve(pevsl_mlp *net, int batch) {
  if (batch <= net->cap) return 0;
  mlp_free_buffers(net);
  int maxd = net->kdim[0];
  for (int l = 0; l < net->layers; l++) maxd = PEVSL_MAX(maxd, net->ndim[l]);
  bool ok = true;
  ok = ok && cudaMalloc(&net->a[0], sizeof(bf16) * (size_t)batch * net->kdim[0]) == cudaSuccess;
  for (int l = 0; l < net->layers && ok; l++) {
    ok = ok && cudaMalloc(&net->z[l], sizeof(float) * (size_t)batch * net->ndim[l]) == cudaSuccess;
    ok = ok && cudaMalloc(&net->a[l + 1], sizeof(bf16) * (size_t)batch * net->ndim[l]) == cudaSuccess;
  }
  ok = ok && cudaMalloc(&net->dz, sizeof(float) * (size_t)batch * maxd) == cudaSuccess;
  ok = ok && cudaMalloc(&net->dzh[0], sizeof(bf16) * (size_t)batch * maxd) == cudaSuccess;
  ok = ok && cudaMalloc(&net->dzh[1], sizeof(bf16) * (size_t)batch * maxd) == cudaSuccess;
  if (!ok) {
    mlp_free_buffers(net);
    return PEVSL_ERR_NOMEM;
  }
  net->cap = batch;
  return 0;
}

/* forward pass on a[0] (already packed); outputs in z[layers-1] */
static int mlp_forward(pevsl_mlp *net, int B) {
  int st = 0;
  for (int l = 0; l < net->layers && !st; l++) {
    const int K = net->kdim[l], N = net->ndim[l];
    const bf16 *W = net->ph + net->woff[l];
    const float *b = net->p + net->boff[l];
    if (l + 1 < net->layers)
      st = gemm<false, true, EPI_BIAS_GELU>(B, N, K, net->a[l], K, W, K, net->z[l], N, b,
                                            net->a[l + 1], N, nullptr, 0);
    else
      st = gemm<false, true, EPI_BIAS>(B, N, K, net->a[l], K, W, K, net->z[l], N, b, nullptr, 0,
                                       nullptr, 0);
  }
  return st;
}

/* loss and gradients into net->g for targets T [B][ldt] (FP32, device) */
static int mlp_backward(pevsl_mlp *net, int B, const float *T, int ldt) {
  Ctx &c = ctx();
  const int L = net->layers;
  int st = 0; /* every entry of g is written below */
  const int NL = net->ndim[L - 1];
  const unsigned gb = grid_for((long)B * NL, 4) > 256 ? 256 : grid_for((long)B * NL, 4);
  if (!st) {
    launch_pdl_block(k_mse, dim3(gb), 256, 0, c.stream, B, NL, net->nout, net->z[L - 1], T, ldt, net->dz,
                     net->dzh[0], net->partials, net->counter, net->loss);
    st = launched("mse");
  }
  int cur = 0;
  for (int l = L - 1; l >= 0 && !st; l--) {
    const int K = net->kdim[l], N = net->ndim[l];
    /* dW_l = dZ_l^T a_l (N x K), db_l = column sums of dZ_l */
    st = gemm<true, false, EPI_STORE>(N, K, B, net->dzh[cur], N, net->a[l], K, net->g + net->woff[l],
                                      K, nullptr, nullptr, 0, net->dz, N, net->g + net->boff[l]);
    if (l == 0 || st) break;
    /* dZ_{l-1} = (dZ_l W_l) * gelu'(z_{l-1}) */
    st = gemm<false, false, EPI_DGELU>(B, K, N, net->dzh[cur], N, net->ph + net->woff[l], K, net->dz,
                                       K, nullptr, net->dzh[1 - cur], K, net->z[l - 1], K);
    cur = 1 - cur;
  }
  return st;
}

extern "C" {

int pEVSL_B200_MlpCreate(pevsl_mlp **out, int nin, int width, int nout, int layers) {
  *out = nullptr;
  if (ensure()) return PEVSL_ERR_CUDA;
  if (nin <= 0 || nout <= 0 || width <= 0 || layers < 1 || layers > 8) return PEVSL_ERR_ARG;
  pevsl_mlp *net = (pevsl_mlp *)calloc(1, sizeof(pevsl_mlp));
  if (!net) return PEVSL_ERR_NOMEM;
  net->nin = nin;
  net->nout = nout;
  net->width = width;
  net->layers = layers;
  long off = 0;
  for (int l = 0; l < layers; l++) {
    net->kdim[l] = pad16(l == 0 ? nin : width);
    net->ndim[l] = pad16(l + 1 == layers ? nout : width);
    net->woff[l] = off;
    off += (long)net->kdim[l] * net->ndim[l];
    net->boff[l] = off;
    off += net->ndim[l];
  }
  net->np = off;
  bool ok = true;
  ok = ok && cudaMalloc(&net->p, sizeof(float) * off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->g, sizeof(float) * off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->m1, sizeof(float) * off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->m2, sizeof(float) * off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->ph, sizeof(bf16) * off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->mask, off) == cudaSuccess;
  ok = ok && cudaMalloc(&net->loss, sizeof(float)) == cudaSuccess;
  ok = ok && cudaMalloc(&net->partials, sizeof(double) * 256) == cudaSuccess;
  ok = ok && cudaMalloc(&net->counter, sizeof(unsigned)) == cudaSuccess;
  if (ok) {
    cudaMemset(net->p, 0, sizeof(float) * off);
    cudaMemset(net->g, 0, sizeof(float) * off);
    cudaMemset(net->m1, 0, sizeof(float) * off);
    cudaMemset(net->m2, 0, sizeof(float) * off);
    cudaMemset(net->ph, 0, sizeof(bf16) * off);
    cudaMemset(net->counter, 0, sizeof(unsigned));
    /* mask of real entries */
    uint8_t *hm = (uint8_t *)calloc((size_t)off, 1);
    if (!hm) ok = false;
    for (int l = 0; l < layers && ok; l++) {
      const int kr = l == 0 ? nin : width, nr = l + 1 == layers ? nout : width;
      for (int n = 0; n < nr; n++) {
        memset(hm + net->woff[l] + (long)n * net->kdim[l], 1, (size_t)kr);
        hm[net->boff[l] + n] = 1;
      }
    }
    ok = ok && cudaMemcpy(net->mask, hm, (size_t)off, cudaMemcpyHostToDevice) == cudaSuccess;
    free(hm);
  }
  if (!ok) {
    pEVSL_B200_MlpFree(net);
    return PEVSL_ERR_NOMEM;
  }
  *out = net;
  return 0;
}

void pEVSL_B200_MlpFree(pevsl_mlp *net) {
  if (!net) return;
  mlp_free_buffers(net);
  cudaFree(net->p);
  cudaFree(net->g);
  cudaFree(net->m1);
  cudaFree(net->m2);
  cudaFree(net->ph);
  cudaFree(net->mask);
  cudaFree(net->loss);
  cudaFree(net->partials);
  cudaFree(net->counter);
  free(net);
}

long pEVSL_B200_MlpParamCount(const pevsl_mlp *net) { return net ? net->np : 0; }

int pEVSL_B200_MlpLayout(const pevsl_mlp *net, int *kdim, int *ndim, long *woff, long *boff) {
  if (!net) return PEVSL_ERR_ARG;
  for (int l = 0; l < net->layers; l++) {
    kdim[l] = net->kdim[l];
    ndim[l] = net->ndim[l];
    woff[l] = net->woff[l];
    boff[l] = net->boff[l];
  }
  return net->layers;
}

/* parameters (FP32 master, the padded layout above) from / to the host;
 * setting them resets the Adam state */
int pEVSL_B200_MlpSetParams(pevsl_mlp *net, const float *host) {
  if (!net || !host) return PEVSL_ERR_ARG;
  if (fail(cudaMemcpy(net->p, host, sizeof(float) * net->np, cudaMemcpyHostToDevice), "MlpSetParams"))
    return PEVSL_ERR_CUDA;
  cudaMemset(net->m1, 0, sizeof(float) * net->np);
  cudaMemset(net->m2, 0, sizeof(float) * net->np);
  net->step = 0;
  k_to_bf16<<<grid_for(net->np, 4), kThreads, 0, ctx().stream>>>(net->np, net->p, net->ph);
  if (launched("to_bf16")) return PEVSL_ERR_CUDA;
  return sync();
}

int pEVSL_B200_MlpGetParams(const pevsl_mlp *net, float *host) {
  if (!net || !host) return PEVSL_ERR_ARG;
  if (sync()) return PEVSL_ERR_CUDA;
  return fail(cudaMemcpy(host, net->p, sizeof(float) * net->np, cudaMemcpyDeviceToHost), "MlpGetParams")
             ? PEVSL_ERR_CUDA
             : 0;
}

/* Y [B][nout] = net(X [B][nin]); X, Y FP32 device (or managed) arrays */
int pEVSL_B200_MlpForward(pevsl_mlp *net, const float *X, float *Y, int B) {
  if (!net || B < 0) return PEVSL_ERR_ARG;
  if (B == 0) return 0;
  if (mlp_reserve(net, B)) return PEVSL_ERR_NOMEM;
  const int K0 = net->kdim[0];
  launch_pdl(k_pack_input, grid_for((long)B * K0, 4), ctx().stream, B, net->nin, K0, X, net->a[0]);
  if (launched("pack_input")) return PEVSL_ERR_CUDA;
  if (mlp_forward(net, B)) return PEVSL_ERR_CUDA;
  const int L = net->layers, NL = net->ndim[L - 1];
  if (fail(cudaMemcpy2DAsync(Y, sizeof(float) * net->nout, net->z[L - 1], sizeof(float) * NL,
                             sizeof(float) * net->nout, B, cudaMemcpyDefault, ctx().stream),
           "MlpForward copy"))
    return PEVSL_ERR_CUDA;
  return sync();
}

/* mean squared error of net(X) against T [B][nout] and its gradient (host
 * FP32, the parameter layout) without updating the weights */
int pEVSL_B200_MlpGradients(pevsl_mlp *net, const float *X, const float *T, int B, float *loss,
                            float *grad_host) {
  if (!net || B <= 0) return PEVSL_ERR_ARG;
  if (mlp_reserve(net, B)) return PEVSL_ERR_NOMEM;
  const int K0 = net->kdim[0];
  launch_pdl(k_pack_input, grid_for((long)B * K0, 4), ctx().stream, B, net->nin, K0, X, net->a[0]);
  if (launched("pack_input")) return PEVSL_ERR_CUDA;
  if (mlp_forward(net, B) || mlp_backward(net, B, T, net->nout)) return PEVSL_ERR_CUDA;
  if (sync()) return PEVSL_ERR_CUDA;
  if (loss && cudaMemcpy(loss, net->loss, sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
    return PEVSL_ERR_CUDA;
  if (grad_host &&
      cudaMemcpy(grad_host, net->g, sizeof(float) * net->np, cudaMemcpyDeviceToHost) != cudaSuccess)
    return PEVSL_ERR_CUDA;
  return 0;
}

/* one Adam step on the batch (X, T); the loss before the step in *loss
 * (may be NULL; reading it synchronises) */
int pEVSL_B200_MlpTrainStep(pevsl_mlp *net, const float *X, const float *T, int B, float lr,
                            float *loss) {
  if (!net || B <= 0) return PEVSL_ERR_ARG;
  if (mlp_reserve(net, B)) return PEVSL_ERR_NOMEM;
  Ctx &c = ctx();
  const int K0 = net->kdim[0];
  launch_pdl(k_pack_input, grid_for((long)B * K0, 4), c.stream, B, net->nin, K0, X, net->a[0]);
  if (launched("pack_input")) return PEVSL_ERR_CUDA;
  if (mlp_forward(net, B) || mlp_backward(net, B, T, net->nout)) return PEVSL_ERR_CUDA;
  net->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)net->step), c2 = 1.f - powf(b2, (float)net->step);
  launch_pdl(k_adam, grid_for(net->np, 4), c.stream, net->np, net->p, net->g, net->m1, net->m2, net->mask,
             net->ph, lr, b1, b2, 1e-8f, c1, c2);
  if (launched("adam")) return PEVSL_ERR_CUDA;
  if (loss) {
    if (memcpy_async(c.hscal + S_TMP0, net->loss, sizeof(float)) || sync()) return PEVSL_ERR_CUDA;
    memcpy(loss, c.hscal + S_TMP0, sizeof(float));
  }
  return 0;
}

}  // extern "C"
