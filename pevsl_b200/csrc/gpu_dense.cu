/*
 * Dense kernels over the Lanczos basis V (n x k, column major, leading
 * dimension ldv), on the FP64 tensor cores (mma.sync m8n8k4 .f64); the
 * Gram-Schmidt passes live in gpu_batch.cu.
 *
 *  - gemm_nn: Ritz vectors U = V(:,0:k) Y (SRC/cheblanNr.c:363-365 does one
 *    GEMV per Ritz vector; here one pass over V serves 64 of them, and up to
 *    four in a kernel without tensor cores).
 *  - gemm_tn: Gram matrices C = V' W of the refinement sweep.
 */
#include <cuda_runtime.h>
#include <float.h>

#include "gpu.cuh"

namespace pv {

/* FP64 tensor-core product (DMMA): D = A B + C for an 8 x 4 tile of A and a
 * 4 x 8 tile of B.  Fragments per lane l: a = A[l / 4][l % 4],
 * b = B[l % 4][l / 4], c/d = C[l / 4][2 (l % 4) + {0, 1}]. */
__device__ __forceinline__ void dmma_8x8x4(double a, double b, double &c0, double &c1) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

/* U = V(:, 0:k) Y on the FP64 tensor cores: a block owns a 64 x 64 tile of
 * U (64 rows, 64 Ritz vectors) and walks k in panels of 16 columns of V,
 * staged in shared memory with the matching 16 rows of Y; each of the 8
 * warps accumulates 8 of the tile's 8 x 8 sub-tiles (warp w: sub-tile rows
 * w, sub-tile columns 0..7).  V is read m / 64 times instead of once per
 * eight Ritz vectors.  (SRC/cheblanNr.c:363-365 forms the Ritz vectors one
 * GEMV each.) */
constexpr int kNnTile = 64, kNnPanel = 16;
__global__ void __launch_bounds__(kThreads)
    k_gemm_nn_dmma(long n, int k, int m, const double *__restrict__ V, long ldv,
                   const double *__restrict__ Y, long ldy, double *__restrict__ U, long ldu) {
  __shared__ double vs[kNnPanel][kNnTile + 1]; /* vs[jj][i] = V[i0 + i, j + jj] */
  __shared__ double ys[kNnPanel][kNnTile + 1]; /* ys[jj][c] = Y[j + jj, c0 + c] */
  const long i0 = (long)blockIdx.x * kNnTile;
  const int c0 = blockIdx.y * kNnTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lr = lane >> 2, lc = lane & 3;
  double acc[8][2];
#pragma unroll
  for (int t = 0; t < 8; t++) acc[t][0] = acc[t][1] = 0.0;
  for (int j = 0; j < k; j += kNnPanel) {
    /* 64 rows x 16 columns of V (a column's 64 rows are contiguous) and 16
     * rows x 64 columns of Y, zero outside */
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int t = threadIdx.x + kThreads * q;
      const int i = t & 63, jj = t >> 6;
      const long row = i0 + i;
      vs[jj][i] = (row < n && j + jj < k) ? V[(size_t)(j + jj) * ldv + row] : 0.0;
      const int c = t >> 4, yj = t & 15;
      ys[yj][c] = (c0 + c < m && j + yj < k) ? Y[(size_t)(c0 + c) * ldy + j + yj] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kNnPanel; kk += 4) {
      const double a = vs[kk + lc][warp * 8 + lr];
#pragma unroll
      for (int t = 0; t < 8; t++) dmma_8x8x4(a, ys[kk + lc][t * 8 + lr], acc[t][0], acc[t][1]);
    }
    __syncthreads();
  }
  const long row = i0 + warp * 8 + lr;
  if (row < n) {
#pragma unroll
    for (int t = 0; t < 8; t++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = c0 + t * 8 + 2 * lc + h;
        if (c < m) U[(size_t)c * ldu + row] = acc[t][h];
      }
  }
}

/* U = V(:, 0:k) Y for one to four columns of Y: a thread per row, Y in shared
 * memory, V read once.  Bound by V's bytes; the DMMA tile pads such products
 * to 64 columns (two Ritz vectors from 50 columns at 10^6 rows: 583 us, here
 * 57 us, 7.3 TB/s with part of V in L2). */
constexpr int kNnSkinnyCols = 1024; /* columns of V per pass over Y in shared memory */
template <int M>
__global__ void __launch_bounds__(kThreads)
    k_gemm_nn_skinny(long n, int k, const double *__restrict__ V, long ldv,
                     const double *__restrict__ Y, long ldy, double *__restrict__ U, long ldu) {
  __shared__ double ys[kNnSkinnyCols][M];
  const long row = blockIdx.x * (long)kThreads + threadIdx.x;
  double acc[M][2] = {};
  for (int j0 = 0; j0 < k; j0 += kNnSkinnyCols) {
    const int kc = k - j0 < kNnSkinnyCols ? k - j0 : kNnSkinnyCols;
    if (j0) __syncthreads();
    for (int t = threadIdx.x; t < kc * M; t += kThreads) ys[t / M][t % M] = Y[(size_t)(t % M) * ldy + j0 + t / M];
    __syncthreads();
    if (row >= n) continue;
    const double *p = V + (size_t)j0 * ldv + row;
    int j = 0;
    for (; j + 7 < kc; j += 8) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; u++) x[u] = __ldg(p + (size_t)(j + u) * ldv);
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int c = 0; c < M; c++) acc[c][u & 1] = fma(x[u], ys[j + u][c], acc[c][u & 1]);
    }
    for (; j < kc; j++) {
      const double x = __ldg(p + (size_t)j * ldv);
#pragma unroll
      for (int c = 0; c < M; c++) acc[c][0] = fma(x, ys[j][c], acc[c][0]);
    }
  }
  if (row < n)
#pragma unroll
    for (int c = 0; c < M; c++) U[(size_t)c * ldu + row] = acc[c][0] + acc[c][1];
}

int gemm_nn(long n, int k, int m, const double *V, long ldv, const double *Y, long ldy, double *U,
            long ldu) {
  if (m <= 0 || n <= 0) return 0;
  if (m <= 4) {
    const unsigned g = (unsigned)((n + kThreads - 1) / kThreads);
    auto kern = m == 1   ? k_gemm_nn_skinny<1>
                : m == 2 ? k_gemm_nn_skinny<2>
                : m == 3 ? k_gemm_nn_skinny<3>
                         : k_gemm_nn_skinny<4>;
    kern<<<g, kThreads, 0, ctx().stream>>>(n, k, V, ldv, Y, ldy, U, ldu);
    return launched("gemm_nn_skinny");
  }
  dim3 g((unsigned)((n + kNnTile - 1) / kNnTile), (unsigned)((m + kNnTile - 1) / kNnTile));
  k_gemm_nn_dmma<<<g, kThreads, 0, ctx().stream>>>(n, k, m, V, ldv, Y, ldy, U, ldu);
  return launched("gemm_nn_dmma");
}

/* C = V' W for tall V (n x k) and W (n x m) on the FP64 tensor cores: a
 * block owns a 64 x 64 tile of C and one chunk of rows; it stages 16 rows of
 * the two 64-column panels in shared memory, and each of the 8 warps
 * accumulates 8 of the tile's 8 x 8 sub-tiles (sub-tile row = warp) with
 * m8n8k4 DMMA over the panel's rows.  Per-chunk tiles go to partial[chunk],
 * then k_gemm_tn_reduce adds them in chunk order (deterministic).  These are
 * the block Gram products of the refinement sweep, the dense counterpart of
 * the reference's GemtvWithWspace (SRC/parvecs.c:117-136). */
constexpr int kTnTile = 64, kTnRows = 16;
__global__ void __launch_bounds__(kThreads)
    k_gemm_tn_partial(long n, int k, int m, const double *__restrict__ V, long ldv,
                      const double *__restrict__ W, long ldw, long rows_per_chunk,
                      double *__restrict__ partial) {
  __shared__ double vs[kTnRows][kTnTile + 1], wsh[kTnRows][kTnTile + 1];
  const int ti = blockIdx.x, tj = blockIdx.y;
  const long r_beg = (long)blockIdx.z * rows_per_chunk;
  const long r_end = r_beg + rows_per_chunk < n ? r_beg + rows_per_chunk : n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lr = lane >> 2, lc = lane & 3;
  double acc[8][2];
#pragma unroll
  for (int t = 0; t < 8; t++) acc[t][0] = acc[t][1] = 0.0;
  for (long r0 = r_beg; r0 < r_end; r0 += kTnRows) {
    /* 16 rows x 64 columns of each panel: thread t loads row t % 16 of
     * columns t / 16 + 16 q (16 consecutive rows of a column per half-warp) */
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = threadIdx.x & 15, c = (threadIdx.x >> 4) + 16 * q;
      const long row = r0 + r;
      const int cv = ti * kTnTile + c, cw = tj * kTnTile + c;
      vs[r][c] = (row < r_end && cv < k) ? V[(size_t)cv * ldv + row] : 0.0;
      wsh[r][c] = (row < r_end && cw < m) ? W[(size_t)cw * ldw + row] : 0.0;
    }
    __syncthreads();
    /* A = V' (rows: columns of V, k: rows of the panel), B = W panel */
#pragma unroll
    for (int kk = 0; kk < kTnRows; kk += 4) {
      const double a = vs[kk + lc][warp * 8 + lr];
#pragma unroll
      for (int t = 0; t < 8; t++) dmma_8x8x4(a, wsh[kk + lc][t * 8 + lr], acc[t][0], acc[t][1]);
    }
    __syncthreads();
  }
  double *out = partial + (size_t)blockIdx.z * (size_t)k * (size_t)m;
  const int ci = ti * kTnTile + warp * 8 + lr;
  if (ci < k) {
#pragma unroll
    for (int t = 0; t < 8; t++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int cj = tj * kTnTile + t * 8 + 2 * lc + h;
        if (cj < m) out[(size_t)cj * k + ci] = acc[t][h];
      }
  }
}
__global__ void k_gemm_tn_reduce(int k, int m, int nchunk, const double *__restrict__ partial,
                                 double *__restrict__ C, long ldc) {
  const long tot = (long)k * m;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < nchunk; c++) s += partial[(size_t)c * tot + t];
    C[(t / k) * ldc + t % k] = s;
  }
}

int gemm_tn(long n, int k, int m, const double *V, long ldv, const double *W, long ldw, double *C,
            long ldc) {
  if (k <= 0 || m <= 0) return 0;
  const int tk = (k + kTnTile - 1) / kTnTile, tm = (m + kTnTile - 1) / kTnTile;
  /* enough row chunks for about four blocks per SM, at least 1024 rows each */
  long nchunk = (4L * 148 + tk * tm - 1) / (tk * tm);
  const long max_chunks = (n + 1023) / 1024;
  if (nchunk > max_chunks) nchunk = max_chunks;
  if (nchunk < 1) nchunk = 1;
  long rows = (n + nchunk - 1) / nchunk;
  rows = (rows + kTnRows - 1) / kTnRows * kTnRows;
  nchunk = n > 0 ? (n + rows - 1) / rows : 1;
  double *part = (double *)ws(WS_GEMM, sizeof(double) * (size_t)nchunk * (size_t)k * (size_t)m);
  if (!part) return PEVSL_ERR_NOMEM;
  dim3 g((unsigned)tk, (unsigned)tm, (unsigned)nchunk);
  k_gemm_tn_partial<<<g, kThreads, 0, ctx().stream>>>(n, k, m, V, ldv, W, ldw, rows, part);
  if (launched("gemm_tn_partial")) return PEVSL_ERR_CUDA;
  k_gemm_tn_reduce<<<grid_for((long)k * m, 1), kThreads, 0, ctx().stream>>>(k, m, (int)nchunk, part,
                                                                            C, ldc);
  return launched("gemm_tn_reduce");
}

/* ---------------------------------------------------------------- small eigenproblem
 * The ends of the spectrum of the projected matrix of a thick restart, and
 * their eigenvectors, by one block in shared memory: Jacobi rotations in the
 * round-robin order, n / 2 disjoint ones at a time (Golub & Van Loan, section
 * 8.5), until the off-diagonal part is below DBL_EPSILON of the norm.  The
 * time is the chain of divisions and square roots and the two barriers of a
 * round; warp 0 computes a round's rotations while the others still rotate
 * the vectors.  50 x 50: 0.57 ms, cyclic rotations on the host 1.3 ms and the
 * vectors' way to the GPU.  (The off-diagonal part is summed itself, not as
 * a difference of sums: over 30 restart matrices of dimension 16 to 59 the
 * largest error of an end is 70 eps against the host's 780, of a vector's last
 * element 69 eps against 7e7.)  Below 16 the host is as fast (it needs n^3, this
 * n rounds of a fixed length), above 112 the two matrices leave shared
 * memory; there the host's runs. */
constexpr int kJacMin = 16, kJacMax = 112, kJacThreads = 1024;

__global__ void __launch_bounds__(kJacThreads)
    k_jacobi_ends(int n, const double *__restrict__ A, int lda, double *Y, double *val) {
  extern __shared__ double sm[];
  const int m = n + (n & 1), h = m / 2, ld = m + 1; /* an odd n gets a zero row */
  double *S = sm, *V = sm + (size_t)m * ld;
  __shared__ double rc[2][kJacMax / 2], rs[2][kJacMax / 2], rt[2][kJacMax / 2];
  __shared__ double red[2][32], lam[kJacMax];
  __shared__ int rp[2][kJacMax / 2], rq[2][kJacMax / 2], rank[kJacMax];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = kJacThreads / 32;
  double big = 0.0;
  for (int i = warp; i < m; i += NW)
    for (int j = lane; j < m; j += 32) {
      const double x = i < n && j < n ? A[(size_t)j * lda + i] : 0.0;
      big = fmax(big, fabs(x));
      S[i * ld + j] = x;
      V[i * ld + j] = i == j ? 1.0 : 0.0;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (lane == 0) red[0][warp] = big;
  __syncthreads();
  for (int w = 0; w < NW; w++) big = fmax(big, red[0][w]);
  /* by a power of two, so that the squares neither overflow nor vanish */
  const int e = big > 0.0 && big <= DBL_MAX ? max(ilogb(big), -1000) : 0;
  for (int i = warp; i < m; i += NW)
    for (int j = lane; j < m; j += 32) S[i * ld + j] = scalbn(S[i * ld + j], -e);
  __syncthreads();
  /* the rotations of round r, by warp 0, into buffer w */
  auto rotations = [&](int r, int w) {
    for (int i = lane; i < h; i += 32) {
      int p = r + i, q = r + m - 1 - i;
      p = i == 0 ? m - 1 : p < m - 1 ? p : p - (m - 1);
      q = q < m - 1 ? q : q - (m - 1);
      const double apq = S[p * ld + q];
      double c = 1.0, t = 0.0;
      if (apq != 0.0) {
        const double theta = (S[q * ld + q] - S[p * ld + p]) / (2.0 * apq);
        t = copysign(1.0, theta) / (fabs(theta) + sqrt(theta * theta + 1.0));
        c = rsqrt(t * t + 1.0);
      }
      rp[w][i] = p;
      rq[w][i] = q;
      rc[w][i] = c;
      rs[w][i] = t * c;
      rt[w][i] = t;
    }
  };
  for (int sweep = 0; sweep < 100; sweep++) {
    double off = 0.0, dia = 0.0;
    for (int i = warp; i < m; i += NW)
      for (int j = lane; j < m; j += 32) {
        const double x = S[i * ld + j];
        if (i == j) dia += x * x; else off += x * x;
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dia += __shfl_xor_sync(0xffffffffu, dia, o);
    }
    if (lane == 0) {
      red[0][warp] = off;
      red[1][warp] = dia;
    }
    if (warp == 0) rotations(0, 0);
    __syncthreads();
    off = dia = 0.0;
    for (int w = 0; w < NW; w++) {
      off += red[0][w];
      dia += red[1][w];
    }
    if (off <= DBL_EPSILON * DBL_EPSILON * (off + dia)) break; /* the same in every thread */
    for (int r = 0; r < m - 1; r++) {
      const int w = r & 1;
      for (int a = warp; a < h; a += NW) {
        const int p = rp[w][a], q = rq[w][a];
        const double ca = rc[w][a], sa = rs[w][a];
        for (int b = lane; b < h; b += 32) {
          if (a == b) {
            const double d = rt[w][a] * S[p * ld + q];
            S[p * ld + p] -= d;
            S[q * ld + q] += d;
            S[p * ld + q] = S[q * ld + p] = 0.0;
          } else {
            /* block (b, a) in the transposed order of operations, so that S
             * stays symmetric to the bit */
            const int u = rp[w][b], v = rq[w][b];
            const double cb = rc[w][b], sb = rs[w][b];
            const double x0 = S[p * ld + u], x3 = S[q * ld + v];
            double x1 = S[p * ld + v], x2 = S[q * ld + u];
            const double cf = a < b ? cb : ca, sf = a < b ? sb : sa;
            const double cg = a < b ? ca : cb, sg = a < b ? sa : sb;
            if (a > b) {
              const double x = x1;
              x1 = x2;
              x2 = x;
            }
            const double y0 = cf * x0 - sf * x1, y1 = sf * x0 + cf * x1;
            const double y2 = cf * x2 - sf * x3, y3 = sf * x2 + cf * x3;
            const double z0 = cg * y0 - sg * y2, z1 = cg * y1 - sg * y3;
            const double z2 = sg * y0 + cg * y2, z3 = sg * y1 + cg * y3;
            S[p * ld + u] = z0;
            S[p * ld + v] = a < b ? z1 : z2;
            S[q * ld + u] = a < b ? z2 : z1;
            S[q * ld + v] = z3;
          }
        }
      }
      __syncthreads();
      /* warp 0 goes on to the next rotations, the others rotate V (row i:
       * eigenvector i) */
      if (warp == 0) {
        if (r + 1 < m - 1) rotations(r + 1, w ^ 1);
      } else {
        for (int a = warp - 1; a < h; a += NW - 1) {
          const double c = rc[w][a], s = rs[w][a];
          double *vp = V + rp[w][a] * ld, *vq = V + rq[w][a] * ld;
          for (int j = lane; j < m; j += 32) {
            const double x = vp[j], y = vq[j];
            vp[j] = c * x - s * y;
            vq[j] = s * x + c * y;
          }
        }
      }
      __syncthreads();
    }
  }
  if (tid < n) lam[tid] = scalbn(S[tid * ld + tid], e);
  if (tid < 6) val[tid] = nan(""); /* stays where a NaN has no rank */
  if (tid < 2 * n) Y[tid] = nan("");
  __syncthreads();
  if (tid < n) {
    const double x = lam[tid];
    int k = 0;
    for (int j = 0; j < n; j++) k += lam[j] < x || (lam[j] == x && j < tid) ? 1 : 0;
    rank[tid] = k;
    if (k == 0) val[0] = x;
    if (k == 1) val[1] = x;
    if (k == n - 2) val[2] = x;
    if (k == n - 1) val[3] = x;
  }
  __syncthreads();
  for (int i = 0; i < n; i++) {
    const int k = rank[i];
    if (k != 0 && k != n - 1) continue;
    if (tid < n) Y[(size_t)(k == 0 ? 0 : n) + tid] = V[i * ld + tid];
    if (tid == 0) val[k == 0 ? 4 : 5] = V[i * ld + n - 1];
  }
}

bool ritz_ends_ok(int n) { return n >= kJacMin && n <= kJacMax; }

int ritz_ends(int n, const double *T, int ldt, double *Y, double *val) {
  if (!ritz_ends_ok(n)) return PEVSL_ERR_ARG;
  const size_t len = (size_t)(n - 1) * (size_t)ldt + (size_t)n;
  double *d = (double *)ws(WS_JAC, sizeof(double) * (len + 8));
  if (!d) return PEVSL_ERR_NOMEM;
  const int m = n + (n & 1);
  const size_t sm = sizeof(double) * 2 * (size_t)m * (size_t)(m + 1);
  static bool attr_done = false;
  if (!attr_done) {
    if (fail(cudaFuncSetAttribute(k_jacobi_ends, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * 2 * kJacMax * (kJacMax + 1))),
             "jacobi attribute"))
      return PEVSL_ERR_CUDA;
    attr_done = true;
  }
  if (memcpy_async(d + 8, T, sizeof(double) * len)) return PEVSL_ERR_CUDA;
  k_jacobi_ends<<<1, kJacThreads, sm, ctx().stream>>>(n, d + 8, ldt, Y, d);
  if (launched("jacobi_ends")) return PEVSL_ERR_CUDA;
  if (memcpy_async(val, d, sizeof(double) * 6)) return PEVSL_ERR_CUDA;
  return sync();
}

}  // namespace pv

extern "C" {

int pEVSL_B200_GemmNN(long n, int k, int m, const double *V, long ldv, const double *Y, long ldy,
                      double *U, long ldu) {
  if (pv::ensure()) return PEVSL_ERR_CUDA;
  if (n < 0 || k < 0 || m < 0 || ldv < n || ldu < n || ldy < k) return PEVSL_ERR_ARG;
  return pv::gemm_nn(n, k, m, V, ldv, Y, ldy, U, ldu);
}

int pEVSL_B200_GemmTN(long n, int k, int m, const double *V, long ldv, const double *W, long ldw,
                      double *C, long ldc) {
  if (pv::ensure()) return PEVSL_ERR_CUDA;
  if (n < 0 || k < 0 || m < 0 || ldv < n || ldw < n || ldc < k) return PEVSL_ERR_ARG;
  return pv::gemm_tn(n, k, m, V, ldv, W, ldw, C, ldc);
}

}  // extern "C"
