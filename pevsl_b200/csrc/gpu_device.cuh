/*
 * Device-side helpers shared by the CUDA modules: fixed-tree warp/block
 * sums, the last-block reduction used by every deterministic reduction, and
 * the Chebyshev recurrence epilogue with explicit rounding so that every
 * kernel that applies it (single vector or batched) gives identical bits.
 */
#ifndef PEVSL_B200_GPU_DEVICE_CUH
#define PEVSL_B200_GPU_DEVICE_CUH

#include <cuda_runtime.h>
#include <stdlib.h>

#include <utility>

#include "gpu.cuh"

namespace pv {

/* Programmatic dependent launch, for the filter-degree kernels first of all.  A degree
 * launched with the stream-serialisation attribute may be scheduled while
 * the previous degree's last blocks still run: its blocks stage the value
 * table in shared memory, then wait (griddepcontrol.wait) until the
 * previous grid has completed and its writes are visible, and only then
 * read a vector.  A block lets the next degree be scheduled
 * (griddepcontrol.launch_dependents) only after its own wait, so the early
 * part of degree k+1 overlaps degree k and nothing older.  What the early
 * part reads, the value table, is written at set-up, followed by a device
 * synchronisation, and never again while the matrix lives.  Without the
 * attribute the wait returns at once.  (Loading the first entries of a row
 * before the wait as well took the one-vector kernel from 32 to 48
 * registers and measured slower.)
 *
 * Such a grid is resident while the one before it still writes, so what an
 * earlier launch wrote is not read-only for its lifetime: vectors, partial
 * sums and scalars are read after the wait, through plain pointers without
 * __restrict__, never through the read-only path (__ldg, const __restrict__),
 * whose loads the compiler may move across the wait.  That path is for what
 * was written at set-up: matrix entries, masks, tables, weights. */
__device__ __forceinline__ void pdl_wait_then_release() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

/* PEVSL_B200_PDL: 1 (default) launches with the attribute, 0 as plain
 * stream-ordered launches */
inline int pdl_mode() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("PEVSL_B200_PDL");
    v = e ? atoi(e) != 0 : 1;
  }
  return v;
}

template <class... KA, class... AA>
void launch_pdl_block(void (*k)(KA...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                      AA &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_mode();
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, std::forward<AA>(args)...);
}

template <class... KA, class... AA>
void launch_pdl(void (*k)(KA...), unsigned grid, cudaStream_t st, AA &&...args) {
  launch_pdl_block(k, dim3(grid), kThreads, 0, st, std::forward<AA>(args)...);
}


__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

/* Sum over the block with a fixed tree; valid in thread 0.  sh needs one
 * double per warp. */
__device__ __forceinline__ double block_sum(double v, double *sh) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  v = warp_sum(v);
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = (int)threadIdx.x < nw ? sh[threadIdx.x] : 0.0;
  if (w == 0) v = warp_sum(v);
  return v;
}

enum Fin { FIN_ID = 0, FIN_SQRT = 1 };

/* Deterministic grid reduction over gridDim.x blocks: this block's partial
 * goes to partials[blockIdx.x]; the last block to arrive (atomic ticket on
 * *counter) adds all partials in block order, applies fin, and returns the
 * total in thread 0 with *is_last set.  *counter is reset for reuse. */
__device__ __forceinline__ double grid_sum(double part, double *partials, unsigned *counter,
                                           int fin, bool *is_last) {
  __shared__ double sh[32];
  __shared__ bool am_last;
  const double s = block_sum(part, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    am_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  *is_last = am_last;
  if (!am_last) return 0.0;
  __threadfence();
  double t = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) t += __ldcg(partials + i);
  t = block_sum(t, sh);
  if (threadIdx.x == 0) *counter = 0;
  return fin == FIN_SQRT ? sqrt(t) : t;
}

/* One Chebyshev filter degree for one row (SRC/chebpol.c:549-559):
 *   w = (A v_k - cc v_k) t - v_{k-1};  y = first ? mu0 v_k + muk w : y + muk w
 * rounded as fma(-cc, x, r) * t, then subtractions and fma for y. */
__device__ __forceinline__ void cheb_update(double r, double x, const double *xm1, double cc,
                                            double t, double mu0, double muk, bool first,
                                            double *w_out, double *y) {
  double w = __dmul_rn(__fma_rn(-cc, x, r), t);
  if (xm1) w = __dsub_rn(w, *xm1);
  *w_out = w;
  *y = first ? __fma_rn(muk, w, __dmul_rn(mu0, x)) : __fma_rn(muk, w, *y);
}

/* cheb_update on values already loaded (xm1 used only when has_m1) */
__device__ __forceinline__ void cheb_update_v(double r, double x, double xm1, bool has_m1,
                                              double cc, double t, double mu0, double muk,
                                              bool first, double yold, double *w_out,
                                              double *y) {
  double w = __dmul_rn(__fma_rn(-cc, x, r), t);
  if (has_m1) w = __dsub_rn(w, xm1);
  *w_out = w;
  *y = first ? __fma_rn(muk, w, __dmul_rn(mu0, x)) : __fma_rn(muk, w, yold);
}

}  // namespace pv

#endif
