/*
 * Batched vector kernels: one launch serves up to kMaxBatch independent
 * vectors (the slices of an interval, advancing in lockstep), selected by a
 * bit mask, each with its own pointers and scalars.  blockIdx.y (or z) is the
 * batch entry; within an entry the work decomposition, and hence every
 * rounding, is the same as for a single vector, so a batched run gives the
 * same bits as running the entries one by one.  The single-vector wrappers
 * of gpu.cuh are these kernels with one entry.
 *
 *   b_dot / b_axpy_dev_nrm2  dots and norms: SRC/parvec.c:123-142
 *   b_gemvT / b_gemv_sub_nrm one CGS pass of CGS_DGKS: SRC/miscla.c:211-240
 *
 * Entries may differ in length (slices of different problems): entry s has
 * length len.n[s] and leading dimension len.ld[s], and is decomposed over
 * exactly the blocks a single-vector launch of that length would use (the
 * grid is as wide as the widest entry; the surplus blocks of a shorter
 * entry leave at once), so its reductions add in the same order.
 *
 * The batched filter degree is cheb_step_batch (gpu_sparse.cu).
 */
#include <cuda_runtime.h>

#include "gpu.cuh"
#include "gpu_device.cuh"

namespace pv {

#define PV_ACTIVE(mask, s) (((mask) >> (s)) & 1u)

/* A Lanczos step is about ten of these launches of 2 to 20 us, each of which
 * needs the one before: they are launched before it ends and wait for it on
 * the device, every block of them, also those without work (a grid that ended
 * before its predecessor would release its successor too early).  Nothing is
 * read before the wait, and what is read right after it through plain
 * pointers.  Plain launches / these: 20 vectors of 40 steps at 41 x 43 x 40
 * 9.8 / 8.3 ms, bounds at 100^3 (200 steps) 35.9 / 32.5 ms. */

/* per-entry decomposition of one launch.  The kernels take this and the
 * pointer tables as __grid_constant__ parameters: indexed by the entry, a
 * plain by-value parameter is copied to local memory by every thread, which
 * cost a skipped pass over 10^6 rows 12-14 us and a dot product 17. */
struct BGeom {
  long n[kMaxBatch];
  long ld[kMaxBatch];
  unsigned nb[kMaxBatch]; /* blocks of entry s (x dimension) */
  int rows[kMaxBatch];    /* gemvT: rows per block of entry s */
};

/* grid_sum over the first nb blocks of the x dimension */
__device__ __forceinline__ double grid_sum_n(double part, double *partials, unsigned *counter,
                                             int fin, unsigned nb, bool *is_last) {
  __shared__ double sh[32];
  __shared__ bool am_last;
  const double s = block_sum(part, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    am_last = atomicAdd(counter, 1u) == nb - 1;
  }
  __syncthreads();
  *is_last = am_last;
  if (!am_last) return 0.0;
  __threadfence();
  double t = 0.0;
  for (unsigned i = threadIdx.x; i < nb; i += blockDim.x) t += __ldcg(partials + i);
  t = block_sum(t, sh);
  if (threadIdx.x == 0) *counter = 0;
  return fin == FIN_SQRT ? sqrt(t) : t;
}

/* ---------------------------------------------------------------- level 1 */

/* Elements t, t + stride, ... of entry s, kLoads of them loaded before any is
 * stored (the vectors may alias as far as the compiler knows, so that a store
 * would hold back the next load); f gets them in order. */
constexpr int kLoads = 4;
template <class L, class F>
__device__ __forceinline__ void each_element(long n, unsigned nb, L load, F f) {
  const long stride = (long)nb * blockDim.x;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += kLoads * stride) {
    decltype(load(i)) e[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; u++)
      if (i + u * stride < n) e[u] = load(i + u * stride);
#pragma unroll
    for (int u = 0; u < kLoads; u++)
      if (i + u * stride < n) f(i + u * stride, e[u]);
  }
}

__global__ void k_b_axpy(const __grid_constant__ BGeom g, const __grid_constant__ CPtrs x,
                         const __grid_constant__ VPtrs y, const __grid_constant__ BScal a,
                         unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || blockIdx.x >= g.nb[s]) return;
  const double c = a.v[s];
  const double *xs = x.p[s];
  double *ys = y.p[s];
  each_element(
      g.n[s], g.nb[s], [&](long i) { return make_double2(xs[i], ys[i]); },
      [&](long i, double2 e) { ys[i] = e.y + c * e.x; });
}

/* x *= 1 / nrm[s], the norm on the device */
__global__ void k_b_scal_inv_dev(const __grid_constant__ BGeom g, const __grid_constant__ VPtrs x,
                                 const double *nrm) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (blockIdx.x >= g.nb[s]) return;
  const double c = 1.0 / nrm[s];
  double *xs = x.p[s];
  each_element(
      g.n[s], g.nb[s], [&](long i) { return xs[i]; }, [&](long i, double e) { xs[i] = e * c; });
}

__global__ void k_b_scal(const __grid_constant__ BGeom g, const __grid_constant__ VPtrs x,
                         const __grid_constant__ BScal a, unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || blockIdx.x >= g.nb[s]) return;
  const double c = a.v[s];
  double *xs = x.p[s];
  each_element(
      g.n[s], g.nb[s], [&](long i) { return xs[i]; }, [&](long i, double e) { xs[i] = e * c; });
}

__global__ void k_b_dot(const __grid_constant__ BGeom g, const __grid_constant__ CPtrs x,
                        const __grid_constant__ CPtrs y, double *partials, unsigned *counters,
                        double *out, int fin, unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || blockIdx.x >= g.nb[s]) return;
  const double *xs = x.p[s], *ys = y.p[s];
  double acc = 0.0;
  each_element(
      g.n[s], g.nb[s], [&](long i) { return make_double2(xs[i], ys[i]); },
      [&](long, double2 e) { acc += e.x * e.y; });
  bool last;
  const double t =
      grid_sum_n(acc, partials + (size_t)s * kMaxRedBlocks, counters + s, fin, g.nb[s], &last);
  if (last && threadIdx.x == 0) out[s] = t;
}

/* y += sign coef[s] x, then z . y: k_b_dot's sums with the update of y in the
 * same pass, 5.2 + 6.7 us as two at 10^6 rows, 8.7 as one. */
__global__ void k_b_axpy_dev_dot(const __grid_constant__ BGeom g, const double *coef, double sign,
                                 const __grid_constant__ CPtrs x, const __grid_constant__ VPtrs y,
                                 const __grid_constant__ CPtrs z, double *partials,
                                 unsigned *counters, double *out) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (blockIdx.x >= g.nb[s]) return;
  const double c = sign * coef[s];
  const double *xs = x.p[s], *zs = z.p[s];
  double *ys = y.p[s];
  double acc = 0.0;
  each_element(
      g.n[s], g.nb[s], [&](long i) { return make_double3(xs[i], ys[i], zs[i]); },
      [&](long i, double3 e) {
        const double v = e.y + c * e.x;
        ys[i] = v;
        acc += e.z * v;
      });
  bool last;
  const double t = grid_sum_n(acc, partials + (size_t)s * kMaxRedBlocks, counters + s, FIN_ID,
                              g.nb[s], &last);
  if (last && threadIdx.x == 0) out[s] = t;
}

/* y -= coef[s] x, then ||y|| */
__global__ void k_b_axpy_dev_nrm2(const __grid_constant__ BGeom g, const double *coef,
                                  const __grid_constant__ CPtrs x, const __grid_constant__ VPtrs y,
                                  double *partials, unsigned *counters, double *nrm,
                                  unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || blockIdx.x >= g.nb[s]) return;
  const double a = -coef[s];
  const double *xs = x.p[s];
  double *ys = y.p[s];
  double acc = 0.0;
  each_element(
      g.n[s], g.nb[s], [&](long i) { return make_double2(xs[i], ys[i]); },
      [&](long i, double2 e) {
        const double v = e.y + a * e.x;
        ys[i] = v;
        acc += v * v;
      });
  bool last;
  const double t = grid_sum_n(acc, partials + (size_t)s * kMaxRedBlocks, counters + s, FIN_SQRT,
                              g.nb[s], &last);
  if (last && threadIdx.x == 0) nrm[s] = t;
}

/* ---------------------------------------------------------------- CGS pass */

constexpr int kGemvtCols = 4; /* columns per warp in gemvT */

static int gemvt_rows(long n) { return n < (1L << 16) ? 256 : 1024; }

/* partial[s][rb][j] = sum_{i in row block rb} V_s[i + j ld_s] v_s[i] (nb[s]
 * row blocks of rows[s] rows; the partials of entry s start at s*pstride) */
__global__ void __launch_bounds__(kThreads)
    k_b_gemvt_partial(const __grid_constant__ BGeom g, int k, const __grid_constant__ CPtrs V, const __grid_constant__ CPtrs v, double *__restrict__ partial,
                      size_t pstride, const int *run, unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.z;
  if (!PV_ACTIVE(mask, s) || (run && run[s] == 0) || blockIdx.x >= g.nb[s]) return;
  extern __shared__ double vsh[];
  const long n = g.n[s], ldv = g.ld[s];
  const int rows = g.rows[s];
  const long r0 = (long)blockIdx.x * rows;
  const int nr = (int)((n - r0) < rows ? (n - r0) : rows);
  const double *vs = v.p[s];
  for (int i = threadIdx.x; i < nr; i += blockDim.x) vsh[i] = vs[r0 + i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int cbase = blockIdx.y * wpb * kGemvtCols;
  double *ps = partial + (size_t)s * pstride;
#pragma unroll
  for (int q = 0; q < kGemvtCols; q++) {
    const int j = cbase + q * wpb + wib;
    if (j >= k) break;
    const double *col = V.p[s] + (size_t)j * ldv + r0;
    double acc = 0.0;
#pragma unroll 8
    for (int i = lane; i < nr; i += 32) acc = fma(col[i], vsh[i], acc);
    acc = warp_sum(acc);
    if (lane == 0) ps[(size_t)blockIdx.x * k + j] = acc;
  }
}

/* w[s*ldw + j] = sum_rb partial[s][rb][j], in row-block order: a block sums
 * 32 columns, all its warps loading tiles of 64 row blocks ahead (registers,
 * then two shared-memory buffers) and warp 0 adding them in order, so that
 * the time is that of the additions (8 cycles each) and not one load latency
 * per few row blocks: 977 row blocks 136 -> 6 us. */
constexpr int kRedTile = 64;
__global__ void __launch_bounds__(kThreads)
    k_b_gemvt_reduce(const __grid_constant__ BGeom g, int k, const double *partial,
                     size_t pstride, double *w, long ldw, const int *run,
                     unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || (run && run[s] == 0)) return;
  __shared__ double sh[2][kRedTile][32];
  constexpr int NW = kThreads / 32, PER = kRedTile / NW;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  const double *ps = partial + (size_t)s * pstride + (j < k ? j : 0);
  const int nrb = (int)g.nb[s];
  double next[PER], acc = 0.0;
  auto fetch = [&](int t) {
#pragma unroll
    for (int q = 0; q < PER; q++) {
      const int b = t + wib * PER + q;
      next[q] = b < nrb ? ps[(size_t)b * k] : 0.0;
    }
  };
  fetch(0);
  for (int t = 0, buf = 0; t < nrb; t += kRedTile, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < PER; q++) sh[buf][wib * PER + q][lane] = next[q];
    __syncthreads();
    fetch(t + kRedTile);
    if (wib == 0) {
      const int m = nrb - t < kRedTile ? nrb - t : kRedTile;
#pragma unroll 16
      for (int r = 0; r < m; r++) acc += sh[buf][r][lane];
    }
  }
  if (wib == 0 && j < k) w[(size_t)s * ldw + j] = acc;
}

/* row . w over k columns: four sums, column j in sum j % 4 (the k % 4 last
 * ones in the first) */
struct RowSums {
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  __device__ __forceinline__ double total() const { return (a0 + a1) + (a2 + a3); }
};

/* v_s -= V_s w_s (thread per row, w_s in shared memory), ||v_s||, and the
 * DGKS flag for the next pass: flag[s] = ||v_s|| <= eta * nrm_old[s].  Bound
 * by the basis' bytes; two rows of a thread run together with eight columns
 * in flight each (64 registers, four blocks per SM): at 10^6 rows, 25 columns
 * on average, 44 us (4.9 TB/s) against 46 for one row with four in flight;
 * 69960 rows (fewer blocks than SMs) 4.1 / 5.7 us; three blocks per SM 46,
 * five (spills) 59 us. */
constexpr int kSubRows = 2;
__global__ void __launch_bounds__(kThreads, 4)
    k_b_gemv_sub_nrm(const __grid_constant__ BGeom g, int k, const __grid_constant__ CPtrs V,
                     const double *w, long ldw, const __grid_constant__ VPtrs v,
                     double *partials, unsigned *counters, double *nrm, const int *run,
                     int *flag_out, double *nrm_old, double eta, unsigned mask) {
  pdl_wait_then_release();
  const int s = blockIdx.y;
  if (!PV_ACTIVE(mask, s) || (run && run[s] == 0) || blockIdx.x >= g.nb[s]) return;
  extern __shared__ double wsh[];
  for (int j = threadIdx.x; j < k; j += blockDim.x) wsh[j] = w[(size_t)s * ldw + j];
  __syncthreads();
  const long n = g.n[s], ldv = g.ld[s], stride = (long)g.nb[s] * blockDim.x;
  const double *Vs = V.p[s];
  double *vs = v.p[s];
  double ss = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += kSubRows * stride) {
    RowSums acc[kSubRows];
    const double *p[kSubRows];
    double old[kSubRows];
#pragma unroll
    for (int q = 0; q < kSubRows; q++) {
      const long r = i + q * stride;
      p[q] = Vs + (r < n ? r : i); /* a row past the end repeats the first, unused */
      old[q] = vs[r < n ? r : i];
    }
    int j = 0;
    for (; j + 7 < k; j += 8) {
      double x[kSubRows][8];
#pragma unroll
      for (int q = 0; q < kSubRows; q++)
#pragma unroll
        for (int u = 0; u < 8; u++) x[q][u] = p[q][(size_t)(j + u) * ldv];
#pragma unroll
      for (int q = 0; q < kSubRows; q++)
#pragma unroll
        for (int u = 0; u < 8; u += 4) {
          acc[q].a0 = fma(x[q][u], wsh[j + u], acc[q].a0);
          acc[q].a1 = fma(x[q][u + 1], wsh[j + u + 1], acc[q].a1);
          acc[q].a2 = fma(x[q][u + 2], wsh[j + u + 2], acc[q].a2);
          acc[q].a3 = fma(x[q][u + 3], wsh[j + u + 3], acc[q].a3);
        }
    }
    for (; j + 3 < k; j += 4) {
#pragma unroll
      for (int q = 0; q < kSubRows; q++) {
        const double x0 = p[q][(size_t)j * ldv], x1 = p[q][(size_t)(j + 1) * ldv];
        const double x2 = p[q][(size_t)(j + 2) * ldv], x3 = p[q][(size_t)(j + 3) * ldv];
        acc[q].a0 = fma(x0, wsh[j], acc[q].a0);
        acc[q].a1 = fma(x1, wsh[j + 1], acc[q].a1);
        acc[q].a2 = fma(x2, wsh[j + 2], acc[q].a2);
        acc[q].a3 = fma(x3, wsh[j + 3], acc[q].a3);
      }
    }
    for (; j < k; j++)
#pragma unroll
      for (int q = 0; q < kSubRows; q++) acc[q].a0 = fma(p[q][(size_t)j * ldv], wsh[j], acc[q].a0);
#pragma unroll
    for (int q = 0; q < kSubRows; q++) {
      const long r = i + q * stride;
      if (r < n) {
        const double nv = old[q] - acc[q].total();
        vs[r] = nv;
        ss = fma(nv, nv, ss);
      }
    }
  }
  bool last;
  const double t = grid_sum_n(ss, partials + (size_t)s * kMaxRedBlocks, counters + s, FIN_SQRT,
                              g.nb[s], &last);
  if (last && threadIdx.x == 0) {
    nrm[s] = t;
    if (flag_out) flag_out[s] = t <= eta * nrm_old[s] ? 1 : 0;
    if (nrm_old) nrm_old[s] = t;
  }
}

/* ---------------------------------------------------------------- host wrappers */

BLen blen_uniform(long n, long ld, int S) {
  BLen l{};
  for (int s = 0; s < S && s < kMaxBatch; s++) {
    l.n[s] = n;
    l.ld[s] = ld;
  }
  return l;
}

/* per-entry geometry: nb[s] = the single-vector grid of entry s; returns
 * the widest, or 0 when no active entry has work */
static unsigned geom(const BLen &len, int S, unsigned mask, int per_thread, BGeom *g) {
  unsigned gx = 0;
  for (int s = 0; s < S; s++) {
    g->n[s] = len.n[s];
    g->ld[s] = len.ld[s];
    g->nb[s] = len.n[s] > 0 ? grid_for(len.n[s], per_thread) : 0;
    g->rows[s] = 0;
    if (PV_ACTIVE(mask, s) && len.n[s] > 0 && g->nb[s] > gx) gx = g->nb[s];
  }
  return gx;
}

int b_axpy(const BLen &len, int S, CPtrs x, VPtrs y, BScal a, unsigned mask) {
  BGeom g;
  const unsigned gx = geom(len, S, mask, 4, &g);
  if (!gx) return 0;
  launch_pdl_block(k_b_axpy, dim3(gx, S), kThreads, 0, ctx().stream, g, x, y, a, mask);
  return launched("b_axpy");
}

int b_axpy_dev_dot(const BLen &len, int S, const double *coef, double sign, CPtrs x, VPtrs y,
                   CPtrs z, double *out) {
  BGeom g;
  unsigned gx = geom(len, S, (1u << S) - 1u, 4, &g);
  for (int s = 0; s < S; s++)
    if (!g.nb[s]) g.nb[s] = 1;
  if (!gx) gx = 1;
  launch_pdl_block(k_b_axpy_dev_dot, dim3(gx, S), kThreads, 0, ctx().stream, g, coef, sign, x, y, z,
                   ctx().red, ctx().cnt, out);
  return launched("b_axpy_dev_dot");
}

int b_scal_inv_dev(const BLen &len, int S, const double *nrm, VPtrs x) {
  BGeom g;
  const unsigned gx = geom(len, S, (1u << S) - 1u, 4, &g);
  if (!gx) return 0;
  launch_pdl_block(k_b_scal_inv_dev, dim3(gx, S), kThreads, 0, ctx().stream, g, x, nrm);
  return launched("b_scal_inv_dev");
}

int b_scal(const BLen &len, int S, VPtrs x, BScal a, unsigned mask) {
  BGeom g;
  const unsigned gx = geom(len, S, mask, 4, &g);
  if (!gx) return 0;
  launch_pdl_block(k_b_scal, dim3(gx, S), kThreads, 0, ctx().stream, g, x, a, mask);
  return launched("b_scal");
}

int b_dot(const BLen &len, int S, CPtrs x, CPtrs y, double *out, int fin, unsigned mask) {
  BGeom g;
  unsigned gx = geom(len, S, mask, 4, &g);
  if (!mask) return 0;
  for (int s = 0; s < S; s++)
    if (!g.nb[s]) g.nb[s] = 1; /* an empty entry still writes its (zero) result */
  if (!gx) gx = 1;
  launch_pdl_block(k_b_dot, dim3(gx, S), kThreads, 0, ctx().stream, g, x, y, ctx().red, ctx().cnt,
                   out, fin, mask);
  return launched("b_dot");
}

int b_axpy_dev_nrm2(const BLen &len, int S, const double *coef, CPtrs x, VPtrs y, double *nrm,
                    unsigned mask) {
  BGeom g;
  unsigned gx = geom(len, S, mask, 4, &g);
  if (!mask) return 0;
  for (int s = 0; s < S; s++)
    if (!g.nb[s]) g.nb[s] = 1;
  if (!gx) gx = 1;
  launch_pdl_block(k_b_axpy_dev_nrm2, dim3(gx, S), kThreads, 0, ctx().stream, g, coef, x, y,
                   ctx().red, ctx().cnt, nrm, mask);
  return launched("b_axpy_dev_nrm2");
}

int b_gemvT(const BLen &len, int S, int k, CPtrs V, CPtrs v, double *w, long ldw, const int *run,
            unsigned mask) {
  if (k <= 0 || !mask) return 0;
  BGeom g;
  geom(len, S, mask, 1, &g);
  unsigned gx = 0;
  int maxrows = 0;
  for (int s = 0; s < S; s++) {
    const int rows = gemvt_rows(len.n[s]);
    g.rows[s] = rows;
    g.nb[s] = len.n[s] > 0 ? (unsigned)((len.n[s] + rows - 1) / rows) : 0;
    if (PV_ACTIVE(mask, s)) {
      gx = g.nb[s] > gx ? g.nb[s] : gx;
      maxrows = rows > maxrows ? rows : maxrows;
    }
  }
  if (!gx) return 0;
  const size_t pstride = (size_t)gx * (size_t)k;
  double *part = (double *)ws(WS_PART, sizeof(double) * (size_t)S * pstride);
  if (!part) return PEVSL_ERR_NOMEM;
  const int cols_per_block = (kThreads / 32) * kGemvtCols;
  dim3 g1(gx, (unsigned)((k + cols_per_block - 1) / cols_per_block), S);
  launch_pdl_block(k_b_gemvt_partial, g1, kThreads, sizeof(double) * maxrows, ctx().stream, g, k, V,
                   v, part, pstride, run, mask);
  if (launched("b_gemvT_partial")) return PEVSL_ERR_CUDA;
  dim3 g2((unsigned)((k + 31) / 32), S);
  launch_pdl_block(k_b_gemvt_reduce, g2, kThreads, 0, ctx().stream, g, k, part, pstride, w, ldw, run,
                   mask);
  return launched("b_gemvT_reduce");
}

int b_gemv_sub_nrm(const BLen &len, int S, int k, CPtrs V, const double *w, long ldw, VPtrs v,
                   double *nrm, const int *run, int *flag_out, double *nrm_old, double eta,
                   unsigned mask) {
  if (!mask) return 0;
  if (k > 12288) return PEVSL_ERR_ARG; /* w must fit in shared memory */
  BGeom g;
  unsigned gx = geom(len, S, mask, 2, &g);
  for (int s = 0; s < S; s++)
    if (!g.nb[s]) g.nb[s] = 1;
  if (!gx) gx = 1;
  const size_t sh = sizeof(double) * (size_t)(k > 0 ? k : 1);
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(k_b_gemv_sub_nrm, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
    attr_done = true;
  }
  launch_pdl_block(k_b_gemv_sub_nrm, dim3(gx, S), kThreads, sh, ctx().stream, g, k, V, w, ldw, v,
                   ctx().red, ctx().cnt, nrm, run, flag_out, nrm_old, eta, mask);
  return launched("b_gemv_sub_nrm");
}

/* ---------------------------------------------------------------- single-vector forms */

int vdot(long n, const double *x, const double *y, double *out) {
  CPtrs a{}, b{};
  a.p[0] = x;
  b.p[0] = y;
  return b_dot(blen_uniform(n, n, 1), 1, a, b, out, FIN_ID, 1u);
}

int vnrm2(long n, const double *x, double *out) {
  CPtrs a{};
  a.p[0] = x;
  return b_dot(blen_uniform(n, n, 1), 1, a, a, out, FIN_SQRT, 1u);
}

int vaxpy_dev_nrm2(long n, const double *coef, const double *x, double *y, double *nrm) {
  CPtrs a{};
  VPtrs b{};
  a.p[0] = x;
  b.p[0] = y;
  return b_axpy_dev_nrm2(blen_uniform(n, n, 1), 1, coef, a, b, nrm, 1u);
}

int gemvT(long n, int k, const double *V, long ldv, const double *v, double *w, const int *run) {
  CPtrs a{}, b{};
  a.p[0] = V;
  b.p[0] = v;
  return b_gemvT(blen_uniform(n, ldv, 1), 1, k, a, b, w, 0, run, 1u);
}

int gemv_sub_nrm(long n, int k, const double *V, long ldv, const double *w, double *v, double *nrm,
                 const int *run, int *flag_out, double *nrm_old, double eta) {
  CPtrs a{};
  VPtrs b{};
  a.p[0] = V;
  b.p[0] = v;
  return b_gemv_sub_nrm(blen_uniform(n, ldv, 1), 1, k, a, w, 0, b, nrm, run, flag_out, nrm_old,
                        eta, 1u);
}

}  // namespace pv
