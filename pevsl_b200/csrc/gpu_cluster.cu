/*
 * Filter applications of small problems, all degrees in one launch.
 *
 * Up to 32768 rows a degree of the Chebyshev recurrence
 * (pEVSL_ChebAv, SRC/chebpol.c:538-568) is a few hundred nanoseconds of
 * work, so a launch per degree spends its time on the launch itself and on
 * the dependent loads row pointer -> entries -> gather through L2.  Here one
 * thread-block cluster applies the whole polynomial to one vector: each of
 * its blocks owns R consecutive rows and keeps, in its shared memory, the
 * entries of those rows and a window of v_k -- its own rows and every column
 * they touch.  A thread keeps v_k, v_{k-1} and the filter sum of its rows in
 * registers.  Per degree it gathers from the window (shared memory, no
 * global load but the coefficient), forms its rows' v_{k+1}, stores them
 * into the next window and, through distributed shared memory, into the
 * windows of the blocks that gather them.
 *
 * The generalized filter (each degree a least-squares B-solve, then the A
 * step) runs the same way with the entries of A and B resident.
 *
 * What bounds it is latency.  A cluster barrier with release and acquire
 * takes about 450 cycles, and a value stored for a neighbour about 0.7 more,
 * so the degrees do not meet there: the values are sent with st.async, which
 * counts their bytes on the receiving block's mbarrier, and a block goes on
 * when its own have arrived (three windows instead of two keep a faster
 * neighbour from overwriting what is still read).  A wait lasts at most a
 * given time (set_cluster_wait); when one runs out its cluster gives up and
 * the call returns PEVSL_ERR_CUDA.  Where some block would
 * send to one that it does not hear from (windows of a matrix without
 * symmetric structure), the cluster barrier ends each degree.
 *
 * Measured per degree, one vector, against a launch per degree (of the CSR
 * kernels, and of the stencil form where a matrix has it): 60 rows 0.38 us,
 * 720 0.57 / 2.5 / 2.1, 7980 rows (19 x 20 x 21) 0.77 / 3.2 / 2.2, 15600 rows
 * 1.03 / 3.2 / 2.2, 2000 rows with 17 scattered entries 1.53 / 4.9; with the
 * barrier 7980 rows 1.0 and 15600 rows 1.17 us.  The generalized filter of two
 * slices at 7980 rows, 25 products per degree (a B-solve of degree 24 and A),
 * 20.6 us per degree against 77 from a launch per product.
 * Past 16384 rows a launch per degree of the stencil form is as fast (26970
 * rows: 2.6 us with the entries in shared memory against 2.2); other matrices
 * run here up to 32768 rows where their entries fit beside the windows.
 *
 * A row's products are formed and added in entry order, unfused, and the
 * recurrence is cheb_update_v's: the results are the bits of the
 * launch-per-degree kernels.  Padding entries multiply a zero slot of the
 * window by zero; adding +0 to a sum that started at +0 changes nothing.
 */
#include <cuda_runtime.h>
#include <limits.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "gpu.cuh"
#include "gpu_device.cuh"

namespace pv {

/* 512 threads: one row each up to 8192 rows, 128 registers for the entries */
constexpr int kClThreads = 512;
constexpr int kClMaxBlocks = 16; /* blocks of a cluster (above 8: opt-in) */

__device__ __forceinline__ double cl_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float cl_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double cl_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float cl_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double cl_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float cl_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double cl_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float cl_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

/* the .aligned forms take one arrival per warp: the warp is converged first */
__device__ __forceinline__ void cl_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

/* the shared-memory address `addr` of this block in block `rank` */
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void cl_store(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
/* the same, counted by the receiving block's mbarrier when it arrives */
__device__ __forceinline__ void cl_send(unsigned addr, double v, unsigned mbar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void cl_send(unsigned addr, float v, unsigned mbar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
               "r"(__float_as_uint(v)), "r"(mbar)
               : "memory");
}

__device__ __forceinline__ unsigned long long cl_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");
  return t;
}

/* a poll for the phase of this parity; HINT: suspended for that many ns at
 * most, 0: for a time that the hardware chooses */
template <int HINT>
__device__ __forceinline__ bool cl_poll(unsigned mbar, unsigned parity) {
  unsigned ok;
  if constexpr (HINT == 0)
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity), "n"(HINT)
        : "memory");
  return ok != 0;
}

/* the word of this block that a block of the cluster sets when it gives up */
__device__ __forceinline__ bool cl_gave_up(unsigned addr) {
  unsigned v;
  asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v != 0;
}

/* the rest of a long wait, by the clock */
__device__ __noinline__ bool cl_wait_long(unsigned mbar, unsigned parity, unsigned long long limit,
                                          unsigned gave_up) {
  const unsigned long long t0 = cl_ns();
  while (!cl_gave_up(gave_up) && cl_ns() - t0 < limit)
    if (cl_poll<10000>(mbar, parity)) return true;
  return false;
}

/* wait for the phase of this parity: false when `limit` ns have passed or
 * another block gave up.  The first poll, which the hardware suspends for a
 * while, is nearly always enough; the rest is out of the way: per degree at
 * 7980 rows 0.83 us, as with a loop of polls alone, 0.85-0.86 with the clock, a
 * hint or the other blocks' word in the loop. */
__device__ __forceinline__ bool cl_wait(unsigned mbar, unsigned parity, unsigned long long limit,
                                        unsigned gave_up) {
  if (cl_poll<0>(mbar, parity)) return true;
  return cl_wait_long(mbar, parity, limit, gave_up);
}

/* one matrix of a job, as the kernel reads it */
struct ClMat {
  const int *ia, *ja;
  const void *a; /* T values */
  int ew;        /* longest row */
};

struct ClJob {
  ClMat A, B; /* B: generalized only */
  const double *x;
  double *y;
  const double *mu, *lmu; /* device coefficients; lmu: of the B-solve */
  double cc, dd, ccB, ddB;
  int n, deg, degB;
};

constexpr int kClMaxJobs = 128; /* jobs of a launch: the table is a kernel parameter (32 KB at most) */
struct ClTable {
  ClJob job[kClMaxJobs];
};
static_assert(sizeof(ClTable) <= 32000, "kernel parameters hold 32764 bytes");

/* A row's entries held by a thread: CW of them in registers, or (CW = 0)
 * in shared memory, entry j of local row i at [j * Rp + i]. */
template <class T, int CW>
struct ClRow {
  unsigned short c[CW];
  T v[CW];
};
template <class T>
struct ClRow<T, 0> {
  int w; /* entries of the row */
};

/* shared-memory entries of one matrix: 16-bit window slots and values */
template <class T>
struct ClEnt {
  unsigned short *slot;
  T *val;
  int Rp;
};

template <class T, int CW>
__device__ __forceinline__ T cl_dot(const ClRow<T, CW> &row, const ClEnt<T> &e, int i,
                                    const T *__restrict__ win) {
  T r = T(0);
  if constexpr (CW > 0) {
#pragma unroll
    for (int j = 0; j < CW; j++) r = cl_add(r, cl_mul(row.v[j], win[row.c[j]]));
  } else {
#pragma unroll 4
    for (int j = 0; j < row.w; j++) {
      const int t = j * e.Rp + i;
      r = cl_add(r, cl_mul(e.val[t], win[e.slot[t]]));
    }
  }
  return r;
}

/* entries of local row i (global row r) into registers or shared memory;
 * lo: the window's first column, Z its zero slot */
template <class T, int CW>
__device__ __forceinline__ void cl_load(ClRow<T, CW> &row, const ClEnt<T> &e, const ClMat &M,
                                        int i, int r, int lo, int Z) {
  const int s = __ldg(M.ia + r), w = __ldg(M.ia + r + 1) - s;
  const T *a = (const T *)M.a;
  if constexpr (CW > 0) {
#pragma unroll
    for (int j = 0; j < CW; j++) {
      const int c = j < w ? __ldg(M.ja + s + j) - lo : Z;
      row.c[j] = (unsigned short)((unsigned)c < (unsigned)Z ? c : Z);
      row.v[j] = j < w ? __ldg(a + s + j) : T(0);
    }
  } else {
    row.w = w;
#pragma unroll 4
    for (int j = 0; j < w; j++) {
      const int t = j * e.Rp + i, c = __ldg(M.ja + s + j) - lo;
      e.slot[t] = (unsigned short)((unsigned)c < (unsigned)Z ? c : Z);
      e.val[t] = __ldg(a + s + j);
    }
  }
}

/* CW: entries of a row in registers (rows of at most CW entries), 0: in
 * shared memory.  RPT rows per thread; Z: slots of a window before its zero
 * slot; Rp: at least R, a multiple of 32. */
template <class T, int RPT, int CW, bool GEN>
__global__ void __launch_bounds__(kClThreads, 1)
    k_filter_cluster(const __grid_constant__ ClTable tab, int Z, int Rp, int nwin, unsigned *err,
                     unsigned long long limit, unsigned withheld) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  __shared__ int s_lo, s_hi, s_tlo[kClMaxBlocks], s_thi[kClMaxBlocks], s_async;
  __shared__ __align__(8) unsigned long long s_mbar[3];
  __shared__ unsigned s_gave_up;
  const unsigned nc = cl_size(), rank = cl_rank();
  const ClJob &J = tab.job[blockIdx.x / nc];
  const int n = J.n, R = (n + (int)nc - 1) / (int)nc, r0 = (int)rank * R;
  const int nloc = n - r0 < 0 ? 0 : (n - r0 < R ? n - r0 : R);
  T *win = (T *)cl_smem; /* nwin windows of Z + 1 slots, rounded up to 16 bytes */
  const int ws1 = (Z + 4) / 4 * 4;
  ClEnt<T> eA{}, eB{};
  {
    unsigned char *p = cl_smem + (size_t)nwin * ws1 * sizeof(T);
    auto take = [&](ClEnt<T> &e, const ClMat &M) {
      e.Rp = Rp;
      if constexpr (CW == 0) {
        e.val = (T *)p;
        p += sizeof(T) * (size_t)Rp * M.ew;
        e.slot = (unsigned short *)p;
        p += sizeof(short) * (size_t)Rp * M.ew;
      }
    };
    take(eA, J.A);
    if constexpr (GEN) take(eB, J.B);
  }
  if (threadIdx.x == 0) {
    s_lo = nloc > 0 ? r0 : 0;
    s_hi = nloc > 0 ? r0 + nloc : 0;
  }
  if ((int)threadIdx.x < nwin) win[(int)threadIdx.x * ws1 + Z] = T(0);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(&s_mbar[i]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_async = nwin == 3;
    s_gave_up = 0;
  }
  __syncthreads();
  /* the window: every column the block's rows touch, and the rows */
  {
    int lo = INT_MAX, hi = INT_MIN;
    auto span = [&](const ClMat &M) {
      if (nloc <= 0) return;
      const int e0 = __ldg(M.ia + r0), e1 = __ldg(M.ia + r0 + nloc);
      for (int t = e0 + (int)threadIdx.x; t < e1; t += kClThreads) {
        const int c = __ldg(M.ja + t);
        lo = min(lo, c);
        hi = max(hi, c + 1);
      }
    };
    span(J.A);
    if constexpr (GEN) span(J.B);
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0 && lo < hi) {
      atomicMin(&s_lo, lo);
      atomicMax(&s_hi, hi);
    }
  }
  cl_barrier();
  if (threadIdx.x < nc) {
    unsigned al = (unsigned)__cvta_generic_to_shared(&s_lo), ah = (unsigned)__cvta_generic_to_shared(&s_hi);
    int lo, hi;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(lo) : "r"(cl_map(al, threadIdx.x)));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(hi) : "r"(cl_map(ah, threadIdx.x)));
    s_tlo[threadIdx.x] = lo;
    s_thi[threadIdx.x] = hi < lo + Z ? hi : lo + Z;
  }
  __syncthreads();
  /* the blocks may run without the cluster barrier when every block that
   * sends to another also receives from it: the same answer in every block */
  if (nwin == 3 && threadIdx.x < nc * nc) {
    auto sends = [&](int from, int to) {
      const int f0 = from * R < n ? from * R : n, f1 = f0 + R < n ? f0 + R : n;
      return f0 < s_thi[to] && f1 > s_tlo[to] && f0 < f1;
    };
    const int a = (int)threadIdx.x / (int)nc, b = (int)threadIdx.x % (int)nc;
    if (a != b && sends(a, b) != sends(b, a)) s_async = 0;
  }
  cl_barrier(); /* also: a block that has no further barrier may end after this one */
  const bool async = s_async != 0;
  const int lo = s_lo, hi = s_hi < lo + Z ? s_hi : lo + Z;
  for (int i = threadIdx.x; i < hi - lo; i += kClThreads) win[i] = (T)J.x[lo + i];
  ClRow<T, CW> rowA[RPT], rowB[GEN ? RPT : 1];
  T x[RPT], xm1[RPT], y[RPT];
  unsigned push[RPT]; /* blocks that gather this row */
#pragma unroll
  for (int q = 0; q < RPT; q++) {
    const int i = q * kClThreads + (int)threadIdx.x, r = r0 + i;
    const bool in = i < nloc;
    push[q] = 0;
    x[q] = xm1[q] = y[q] = T(0);
    if (in) {
      cl_load<T, CW>(rowA[q], eA, J.A, i, r, lo, Z);
      if constexpr (GEN) cl_load<T, CW>(rowB[q], eB, J.B, i, r, lo, Z);
      x[q] = (T)J.x[r];
      for (unsigned b = 0; b < nc; b++)
        if (b != rank && r >= s_tlo[b] && r < s_thi[b]) push[q] |= 1u << b;
    }
  }
  __syncthreads();
  int cur = 0; /* the window read */
  auto next = [&]() { return cur + 1 == nwin ? 0 : cur + 1; };
  /* the value of row q into the next window, here and where it is gathered */
  auto publish = [&](int q, T v) {
    const int r = r0 + q * kClThreads + (int)threadIdx.x, to = next();
    T *w = win + to * ws1;
    w[r - lo] = v;
    unsigned m = push[q];
    const unsigned base = (unsigned)__cvta_generic_to_shared(w);
    const unsigned mb = (unsigned)__cvta_generic_to_shared(&s_mbar[to]);
    while (m) {
      const int b = __ffs((int)m) - 1;
      m &= m - 1;
      const unsigned at = cl_map(base + (unsigned)(r - s_tlo[b]) * (unsigned)sizeof(T), (unsigned)b);
      if (async)
        cl_send(at, v, cl_map(mb, (unsigned)b));
      else
        cl_store(at, v);
    }
  };
  /* The end of a step: the next window is complete and becomes the one read.
   * With the barrier, every block's.  Without: this block's rows (the block
   * barrier) and the values sent to it (its mbarrier counts their bytes).  A
   * block that is a step ahead writes the window after that one, which the
   * slower block read two steps ago: its own values for the step before, which
   * the faster one waited for, were sent past the barrier that ended those
   * reads.  False when a wait ran out. */
  const unsigned rx = (unsigned)(hi - lo - nloc) * (unsigned)sizeof(T);
  unsigned parity = 0; /* bit i: of window i's mbarrier */
  const unsigned gave_up = (unsigned)__cvta_generic_to_shared(&s_gave_up);
  auto arm = [&]() {
    if (async && rx && threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(&s_mbar[next()])),
                   "r"(rx + withheld)
                   : "memory");
  };
  auto advance = [&]() -> bool {
    cur = next();
    if (!async) {
      cl_barrier();
      return true;
    }
    bool ok = true;
    if (rx) {
      ok = cl_wait((unsigned)__cvta_generic_to_shared(&s_mbar[cur]), (parity >> cur) & 1u, limit,
                   gave_up);
      parity ^= 1u << cur;
    }
    return !__syncthreads_or(!ok);
  };
  bool ok = true;
  const T cc = (T)J.cc, t1 = (T)(1.0 / J.dd), t2 = (T)(2.0 / J.dd), mu0 = (T)__ldg(J.mu);
  if constexpr (!GEN) {
    T muk = (T)__ldg(J.mu + 1);
    for (int k = 1; k <= J.deg && ok; k++) {
      if (k < J.deg) arm();
      const T mnext = k < J.deg ? (T)__ldg(J.mu + k + 1) : T(0);
      const T *w = win + cur * ws1;
#pragma unroll
      for (int q = 0; q < RPT; q++) {
        const int i = q * kClThreads + (int)threadIdx.x;
        if (i >= nloc) continue;
        const T r = cl_dot<T, CW>(rowA[q], eA, i, w);
        T v = cl_mul(cl_fma(-cc, x[q], r), k == 1 ? t1 : t2);
        if (k > 1) v = cl_sub(v, xm1[q]);
        y[q] = k == 1 ? cl_fma(muk, v, cl_mul(mu0, x[q])) : cl_fma(muk, v, y[q]);
        xm1[q] = x[q];
        x[q] = v;
        if (k < J.deg) publish(q, v);
      }
      muk = mnext;
      if (k < J.deg) ok = advance();
    }
    if (J.deg == 1 && !async) cl_barrier(); /* y may be x: every block has read it */
  } else {
    const T ccB = (T)J.ccB, b1 = (T)(1.0 / J.ddB), b2 = (T)(2.0 / J.ddB), lmu0 = (T)__ldg(J.lmu);
    T l[RPT], lm1[RPT], s[RPT];
    for (int k = 1; k <= J.deg && ok; k++) {
      const T muk = (T)__ldg(J.mu + k);
      /* s = the least-squares B^{-1} of v_k (in the window) */
      T lk = (T)__ldg(J.lmu + 1);
      for (int j = 1; j <= J.degB && ok; j++) {
        arm();
        const T lnext = j < J.degB ? (T)__ldg(J.lmu + j + 1) : T(0);
        const T *w = win + cur * ws1;
#pragma unroll
        for (int q = 0; q < RPT; q++) {
          const int i = q * kClThreads + (int)threadIdx.x;
          if (i >= nloc) continue;
          if (j == 1) l[q] = x[q];
          const T r = cl_dot<T, CW>(rowB[q], eB, i, w);
          T v = cl_mul(cl_fma(-ccB, l[q], r), j == 1 ? b1 : b2);
          if (j > 1) v = cl_sub(v, lm1[q]);
          s[q] = j == 1 ? cl_fma(lk, v, cl_mul(lmu0, l[q])) : cl_fma(lk, v, s[q]);
          lm1[q] = l[q];
          l[q] = v;
          publish(q, j < J.degB ? v : s[q]);
        }
        lk = lnext;
        ok = advance();
      }
      if (!ok) break;
      if (k < J.deg) arm();
      const T *w = win + cur * ws1;
#pragma unroll
      for (int q = 0; q < RPT; q++) {
        const int i = q * kClThreads + (int)threadIdx.x;
        if (i >= nloc) continue;
        const T r = cl_dot<T, CW>(rowA[q], eA, i, w);
        T v = cl_mul(cl_fma(-cc, x[q], r), k == 1 ? t1 : t2);
        if (k > 1) v = cl_sub(v, xm1[q]);
        y[q] = k == 1 ? cl_fma(muk, v, cl_mul(mu0, x[q])) : cl_fma(muk, v, y[q]);
        xm1[q] = x[q];
        x[q] = v;
        if (k < J.deg) publish(q, v);
      }
      if (k < J.deg) ok = advance();
    }
  }
  if (async) {
    /* no block ends while another may still write its windows, nor writes a
     * result over an input that another has yet to read */
    if (!ok && threadIdx.x < nc)
      asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(gave_up, threadIdx.x)),
                   "r"(1)
                   : "memory");
    cl_barrier();
    if (cl_gave_up(gave_up)) {
      /* the same in every block.  Nobody sends any more; values sent before
       * take a microsecond or two, and nobody waits for them: give them 100 */
      if (threadIdx.x == 0) {
        if (rank == 0) atomicExch_system(err, 1u);
        for (const unsigned long long t0 = cl_ns(); cl_ns() - t0 < 100000;) __nanosleep(1000);
      }
      ok = false;
      cl_barrier();
    }
  }
#pragma unroll
  for (int q = 0; q < RPT; q++) {
    const int i = q * kClThreads + (int)threadIdx.x;
    if (i < nloc) J.y[r0 + i] = ok ? (double)y[q] : nan("");
  }
}

/* ---------------------------------------------------------------- host side */

/* shape of a launch: blocks per cluster, rows per thread, row entries in
 * registers (0: shared memory), window slots, rows and shared memory */
struct ClShape {
  int nc, rpt, cw, Z, Rp, nwin;
  size_t smem;
};

constexpr size_t kClSmem = 230000; /* dynamic shared memory of a block, of 232448 bytes */
constexpr int kClRegs = 7;         /* entries of a row that fit a thread's registers */

/* the shape that serves all ne jobs with nc blocks per cluster; false when
 * a job's rows do not fit */
static bool cl_shape(int ne, const ClusterJob *jobs, bool fp32, int nc, ClShape *s) {
  const size_t T = fp32 ? 4 : 8;
  int rmax = 0, zmax = 0, ew = 0, ewsum = 0;
  for (int e = 0; e < ne; e++) {
    const pevsl_devcsr *A = jobs[e].A, *B = jobs[e].B;
    const int n = A->nrows, R = (n + nc - 1) / nc;
    const int kl = B ? std::max(A->band_lo, B->band_lo) : A->band_lo;
    const int ku = B ? std::max(A->band_hi, B->band_hi) : A->band_hi;
    rmax = std::max(rmax, R);
    zmax = std::max(zmax, (int)std::min<long>(n, (long)R + kl + ku));
    ew = std::max(ew, std::max(A->max_row_nnz, B ? B->max_row_nnz : 0));
    ewsum = std::max(ewsum, A->max_row_nnz + (B ? B->max_row_nnz : 0));
  }
  s->nc = nc;
  s->Z = zmax;
  s->Rp = (rmax + 31) / 32 * 32;
  s->rpt = 1;
  while (s->rpt * kClThreads < rmax) s->rpt *= 2;
  if (s->rpt > 4 || zmax > 65535) return false;
  const size_t win = T * (size_t)(zmax + 4);
  s->nwin = 2;
  s->smem = 2 * win;
  s->cw = ew <= kClRegs && s->rpt <= (jobs[0].B ? 1 : 2) ? kClRegs : 0;
  if (!s->cw) s->smem += (T + 2) * (size_t)s->Rp * (size_t)ewsum;
  if (s->smem + win <= kClSmem) {
    s->nwin = 3;
    s->smem += win;
  }
  return s->smem <= kClSmem;
}

template <class T, bool GEN>
static const void *cl_kernel(const ClShape &s) {
  if (s.cw) {
    if constexpr (!GEN)
      if (s.rpt == 2) return (const void *)k_filter_cluster<T, 2, kClRegs, GEN>;
    return (const void *)k_filter_cluster<T, 1, kClRegs, GEN>;
  }
  return s.rpt == 1   ? (const void *)k_filter_cluster<T, 1, 0, GEN>
         : s.rpt == 2 ? (const void *)k_filter_cluster<T, 2, 0, GEN>
                      : (const void *)k_filter_cluster<T, 4, 0, GEN>;
}

static void cl_config(const ClShape &s, int ne, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at) {
  memset(cfg, 0, sizeof *cfg);
  cfg->gridDim = dim3((unsigned)(ne * s.nc));
  cfg->blockDim = dim3(kClThreads);
  cfg->dynamicSmemBytes = s.smem;
  cfg->stream = ctx().stream;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)s.nc;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

static int cl_attributes(const void *k, const ClShape &s) {
  if (fail(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem),
           "cudaFuncSetAttribute") ||
      (s.nc > 8 && fail(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
                        "cudaFuncSetAttribute")))
    return PEVSL_ERR_CUDA;
  return 0;
}

/* clusters of nc blocks (one block per SM) that run at the same time; on a
 * B200 148, 74, 33, 15 and 7 for 1, 2, 4, 8 and 16 blocks */
static int cl_resident(int nc) {
  static int have[kClMaxBlocks + 1] = {0}; /* 0: not asked yet, -1: none */
  if (!have[nc]) {
    ClShape s{nc, 1, kClRegs, 0, 0, 2, kClSmem};
    const void *k = cl_kernel<double, false>(s);
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg;
    cl_config(s, 1, &cfg, &at);
    int m = 0;
    if (cl_attributes(k, s) || cudaOccupancyMaxActiveClusters(&m, k, &cfg) != cudaSuccess) {
      cudaGetLastError();
      m = 0;
    }
    have[nc] = m > 0 ? m : -1;
  }
  return have[nc];
}

/* The shape for ne jobs in one launch: the one whose waves of clusters take
 * the least time by the measured cost of a step (us): the chain of dependent
 * operations and the wait for the other blocks, 0.4 ns per row of a block
 * (1.8 ns with the entries in shared memory) and 60 ns per value that a row
 * sends (the window beyond a block's own rows, over these). */
static bool cl_choose(int ne, const ClusterJob *jobs, bool fp32, ClShape *best) {
  double tbest = 0.0;
  for (int nc = 1; nc <= kClMaxBlocks; nc *= 2) {
    ClShape s;
    if (!cl_shape(ne, jobs, fp32, nc, &s)) continue;
    const int m = cl_resident(nc);
    if (m <= 0) continue;
    const double step = (nc > 1 ? 0.43 : 0.3) + (s.cw ? 0.0 : 0.6) + (s.cw ? 0.0004 : 0.0018) * s.Rp +
                        0.06 * (s.Z - s.Rp > 0 ? (double)(s.Z - s.Rp) / s.Rp : 0.0);
    const double t = ((ne + m - 1) / m) * step;
    if (tbest == 0.0 || t < tbest) {
      tbest = t;
      *best = s;
    }
  }
  return tbest > 0.0;
}

bool cluster_filter_ok(const pevsl_devcsr *A, const pevsl_devcsr *B, bool fp32) {
  if (!A || A->lanes != 0 || A->nrows < 1 || A->nrows > kClusterMaxRows || A->nrows != A->ncols)
    return false;
  if (B && (B->lanes != 0 || B->nrows != A->nrows || B->ncols != A->nrows)) return false;
  ClusterJob J{};
  J.A = A;
  J.B = B;
  ClShape s;
  if (!cl_choose(1, &J, fp32, &s)) return false;
  /* A matrix in the stencil form takes 2.1 us per launched degree, less than a
   * cluster with more than two rows per thread.  A general one is not slower
   * here where its entries fit, k_csr_ahead included (us per degree, cluster /
   * launched, one vector and four in lockstep): 16000 rows of 9 entries 2.81 /
   * 2.94 and 2.90 / 4.78, 24000 of 5 2.96 / 3.12 and 2.93 / 4.54, 32000 of 3 2.86
   * / 2.74 and 2.82 / 3.89, 12000 of 13 2.89 / 3.11 and 2.85 / 5.01. */
  return B || fp32 || !A->smask || s.rpt <= 2;
}

/* two seconds: a step's wait is for neighbours that run at the same time */
constexpr unsigned long long kClWaitNs = 2000000000ull;
static unsigned long long g_cluster_wait = kClWaitNs;
static unsigned g_cluster_withheld = 0;

void set_cluster_wait(long us) {
  g_cluster_wait = us < 0 ? kClWaitNs : 1000ull * (unsigned long long)us;
}

void withhold_cluster_values(bool on) { g_cluster_withheld = on ? 8 : 0; }

int cluster_filter(int ne, const ClusterJob *jobs, bool fp32) {
  if (ne <= 0) return 0;
  const bool gen = jobs[0].B != nullptr;
  /* the longest jobs first; one launch for as many as one shape serves */
  std::vector<ClusterJob> L(jobs, jobs + ne);
  std::stable_sort(L.begin(), L.end(), [](const ClusterJob &a, const ClusterJob &b) {
    return (long)a.deg * a.A->nrows > (long)b.deg * b.A->nrows;
  });
  static ClTable tab; /* host staging: the launch copies it */
  for (int first = 0, nb = 0; first < ne; first += nb) {
    ClShape s;
    nb = std::min(ne - first, kClMaxJobs);
    while (nb > 0 && !cl_choose(nb, &L[(size_t)first], fp32, &s)) nb--;
    if (nb <= 0) return PEVSL_ERR_ARG;
    for (int e = 0; e < nb; e++) {
      const ClusterJob &C = L[(size_t)(first + e)];
      auto mat = [&](const pevsl_devcsr *M) {
        return ClMat{M->ia, M->ja, fp32 ? (const void *)M->a32 : (const void *)M->a, M->max_row_nnz};
      };
      tab.job[e] = ClJob{mat(C.A), gen ? mat(C.B) : ClMat{}, C.x, C.y, C.mu, C.lmu, C.cc, C.dd,
                         C.ccB, C.ddB, C.A->nrows, C.deg, C.degB};
    }
    const void *k = gen    ? cl_kernel<double, true>(s)
                    : fp32 ? cl_kernel<float, false>(s)
                           : cl_kernel<double, false>(s);
    if (cl_attributes(k, s)) return PEVSL_ERR_CUDA;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg;
    cl_config(s, nb, &cfg, &at);
    unsigned *err = ctx().cl_err;
    void *args[] = {(void *)&tab,    (void *)&s.Z, (void *)&s.Rp,
                    (void *)&s.nwin, (void *)&err, (void *)&g_cluster_wait,
                    (void *)&g_cluster_withheld};
    if (fail(cudaLaunchKernelExC(&cfg, k, args), "filter_cluster")) return PEVSL_ERR_CUDA;
    if (launched("filter_cluster")) return PEVSL_ERR_CUDA;
  }
  return 0;
}

}  // namespace pv
