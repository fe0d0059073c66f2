/*
 * pevsl-b200 device runtime shared by the CUDA modules: the per-process GPU
 * context (one stream, reduction scratch, device scalars, cached
 * workspaces), launch accounting, and the host-callable wrappers of the
 * kernels.  Everything is enqueued on the context stream; wrappers return 0
 * or PEVSL_ERR_CUDA and never synchronise unless their name says so.
 */
#ifndef PEVSL_B200_GPU_CUH
#define PEVSL_B200_GPU_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace pv {

constexpr int kThreads = 256;      /* block size of the streaming kernels      */
constexpr int kMaxRedBlocks = 1184; /* 8 x 148 SMs: partial sums per reduction */
constexpr int kMaxBatch = 16;       /* entries of one batched launch            */
constexpr int kMaxEntries = 256;    /* entries of one lockstep group / persistent filter */

/* per-entry pointers / scalars of a batched launch (kernel parameters) */
struct VPtrs {
  double *p[kMaxBatch];
};
struct CPtrs {
  const double *p[kMaxBatch];
};
struct BScal {
  double v[kMaxBatch];
};
/* per-entry filter data of a batched filter degree */
struct BatchParams {
  unsigned mask;          /* active entries */
  int deg[kMaxBatch];     /* filter degree of each entry */
  double cc[kMaxBatch];   /* centre of the spectrum bounds */
  double t1[kMaxBatch];   /* 1 / dd */
  double t2[kMaxBatch];   /* 2 / dd */
};

/* device scalar slots (doubles) */
enum Slot {
  S_ALPHA = 0,
  S_BETA = 1,
  S_NRM0 = 2,
  S_NRM = 3,
  S_TMP0 = 4,
  S_TMP1 = 5,
  S_TMP2 = 6,
  S_TMP3 = 7,
  S_COUNT = 64
};
/* device int flag slots */
enum Flag { F_PASS2 = 0, F_COUNT = 16 };
/* cached workspace slots */
enum Ws {
  WS_BASIS = 0, /* Lanczos basis                              */
  WS_CHEB,      /* three recurrence vectors                   */
  WS_VEC,       /* misc vectors                               */
  WS_KPM,       /* KPM blocks                                 */
  WS_MOM,       /* KPM moments                                */
  WS_PART,      /* CGS partial products                       */
  WS_SMALL,     /* small coefficient arrays                   */
  WS_RITZ,      /* Ritz vectors                               */
  WS_RITZ2,     /* A * Ritz vectors                           */
  WS_REF1,      /* refinement sweep: A P                      */
  WS_REF2,      /* refinement sweep: refined vectors          */
  WS_H,         /* refinement sweep: small projected matrices */
  WS_GEMM,      /* gemm_tn partial tiles                      */
  WS_FILT,      /* batched filter work vectors                */
  WS_MU,        /* filter coefficients on the device          */
  WS_GROUP,     /* per-entry coefficient vectors of a group   */
  WS_ZBASIS,    /* generalized problem: Z = B V               */
  WS_GEN,       /* generalized problem: filter / KPM vectors  */
  WS_IL,        /* interleaved filter: three n x S blocks     */
  WS_ILMU,      /* interleaved filter: per-degree coefficients */
  WS_CLMU,      /* cluster filter: one polynomial's coefficients */
  WS_LAN,       /* Lanczos runs: alpha and beta of every step, CGS coefficients */
  WS_TUNE,      /* scratch vectors of the autotuner (its own: a tuning may come
                   between other uses)                        */
  WS_JAC,       /* projected matrix of a thick restart       */
  WS_LANV,      /* Lanczos DOS: the start vectors of a group */
  WS_COUNT
};

constexpr int kSideStreams = 3;
struct Ctx {
  bool ready = false;
  int device = 0;
  int sms = 148;
  cudaStream_t stream = nullptr;
  double *red = nullptr;       /* kMaxRedBlocks * 64 partial sums */
  unsigned *cnt = nullptr;     /* last-block counters, kept at 0  */
  double *dscal = nullptr;     /* S_COUNT device scalars          */
  double *hscal = nullptr;     /* pinned mirror of dscal          */
  int *dflag = nullptr;        /* F_COUNT device flags            */
  double *gscal = nullptr;     /* 4 * kMaxEntries per-entry device scalars */
  double *hgscal = nullptr;    /* pinned mirror of gscal          */
  int *gflag = nullptr;        /* kMaxEntries per-entry device flags       */
  void *htab = nullptr;        /* pinned staging of the persistent filter table, kTabSlots slots */
  void *dtab = nullptr;        /* device copies of those tables   */
  cudaEvent_t tab_ev[4] = {};  /* copy of slot i done             */
  int tab_next = 0;
  unsigned *bar = nullptr;     /* grid barrier: count, generation, error   */
  cudaMemPool_t pool = nullptr; /* matrices (pool_alloc)          */
  cudaStream_t side[kSideStreams] = {}; /* branches of captured graphs */
  cudaEvent_t side_ev[kSideStreams + 1] = {};
  unsigned *cl_err = nullptr;  /* pinned: a wait of a cluster launch ran out */
  void *ws[WS_COUNT] = {};
  size_t wsz[WS_COUNT] = {};
  uint64_t launches = 0;
  int sticky_error = 0;
};

Ctx &ctx();
int ensure();                 /* initialise the context; 0 or PEVSL_ERR_CUDA */
int fail(cudaError_t e, const char *what);
int launched(const char *what); /* count a launch and check for errors */
/* point the L2 persisting window at [base, base+bytes) if enabled */
void l2_window(const void *base, size_t bytes);
int sync();
void *ws(int slot, size_t bytes);
/* the same without a report when there is no memory (what the slot held is
 * gone then); ws_free gives a slot back */
void *ws_try(int slot, size_t bytes);
void ws_free(int slot);
/* device memory of matrices, in order on the context stream, from a pool that
 * keeps up to 64 MB of freed memory (pEVSL_B200_ReleaseWorkspace gives it
 * back); NULL when there is none */
void *pool_alloc(size_t bytes);
void pool_free(void *p);
int memcpy_async(void *dst, const void *src, size_t bytes);
/* scalar slots: copy device slots [first, first+count) to the pinned mirror
 * and wait; returns pointer into the mirror or NULL */
const double *fetch_scalars(int first, int count);

inline unsigned grid_for(long n, int per_thread = 1) {
  long b = (n + (long)kThreads * per_thread - 1) / ((long)kThreads * per_thread);
  if (b < 1) b = 1;
  if (b > kMaxRedBlocks) b = kMaxRedBlocks;
  return (unsigned)b;
}

/* ---------------------------------------------------------------- BLAS1 */
int vfill(double *x, long n, double v);
int vcopy(const double *x, double *y, long n);
int vscal(double *x, long n, double a);
int vaxpy(long n, double a, const double *x, double *y);
/* *out = <x, y> (deterministic); out in device memory */
int vdot(long n, const double *x, const double *y, double *out);
/* *out = ||x|| */
int vnrm2(long n, const double *x, double *out);
/* *out = sum x */
int vsum(long n, const double *x, double *out);
/* y -= (*coef) x  then  *nrm = ||y||  (one pass) */
int vaxpy_dev_nrm2(long n, const double *coef, const double *x, double *y, double *nrm);
/* out[c] = <X[:,c], Y[:,c]> for c < m, column-major with leading dims */
int vdot_cols(long n, int m, const double *X, long ldx, const double *Y, long ldy, double *out);
/* X[:,c] *= s[c] for c < m (s device) */
int vscal_cols(long n, int m, double *X, long ldx, const double *s);
/* Y[:,c] -= lam[c] X[:,c] (lam device) */
int vaxpy_cols(long n, int m, const double *lam, const double *X, long ldx, double *Y, long ldy);

/* ---------------------------------------------------------------- random */
/* Philox Gaussian draws m0 .. m0+nv-1 into columns of X: X[i*rs + c*cs]. */
int rand_gauss(double *X, long n, int nv, long rs, long cs, uint64_t seed, uint64_t m0);

/* ---------------------------------------------------------------- sparse */
int spmv(const pevsl_devcsr *A, const double *x, double *y);
/* y_s = A x_s for S <= kMaxBatch vectors, each as spmv gives it */
int spmv_batch(const pevsl_devcsr *A, int S, CPtrs x, VPtrs y);
/* One degree of the Chebyshev filter recurrence (fused SpMV):
 *   w = ((A vk - cc vk) * t) - vkm1   (vkm1 may be NULL)
 *   vkp1 = w;  y = first ? mu0 * vk + muk * w : y + muk * w            */
int cheb_step(const pevsl_devcsr *A, const double *vk, const double *vkm1, double *vkp1,
              double *y, double cc, double t, double mu0, double muk, int first);
/* cheb_step with a deferred sum, for matrices where cheb_defers: degree k
 * adds the terms of the last ny degrees (0..3) to y as cheb_step_il_y does;
 * mu on the host */
bool cheb_defers(const pevsl_devcsr *A);
int cheb_step_y(const pevsl_devcsr *A, const double *vk, const double *vkm1, double *vkp1, double *y,
                double cc, double t, const double *mu, int k, int ny, int fresh);
/* terms that degree k of a sum up to degree maxdeg adds to y when the last
 * update was at degree lastw (0: none yet) and D degrees share an update:
 * the first update at degree min(D, 2), the last at maxdeg */
inline int deferred_terms(int k, int lastw, int maxdeg, int D) {
  const int span = lastw == 0 ? (D < 2 ? D : 2) : D;
  return (k == maxdeg || k - lastw == span) ? k - lastw : 0;
}
/* y = sum_{k <= m} mu[k] T_k((A - cc)/dd) v, m >= 1: the degrees of one
 * vector, the sum deferred where cheb_defers; b0, b1: n doubles each.
 * *bytes (if given) receives the algorithmic bytes. */
int cheb_degrees(const pevsl_devcsr *A, const double *mu, int m, double cc, double dd,
                 const double *v, double *y, double *b0, double *b1, double *bytes);
/* The degree of the generalized filter (SRC/chebpol.c:543-546): the SpMV
 * reads x = B^{-1} vk, the recurrence uses vk; tmp (n doubles) is used
 * only by the row-group kernels. */
int cheb_step_x(const pevsl_devcsr *A, const double *x, const double *vk, const double *vkm1,
                double *vkp1, double *y, double cc, double t, double mu0, double muk, int first,
                double *tmp);
/* Fused steps of the Chebyshev iterations for B x = b
 * (EXTERNAL/ITERSOL/chebiter.c): first kind r = b - B x; p = bet p + r;
 * xnew = x + alp p.  Second kind x += d; r -= B d; dnew = c1 d + c2 r. */
int chebiter1_step(const pevsl_devcsr *B, const double *b, const double *x, double *p, double *xnew,
                   double bet, double alp, double *tmp);
int chebiter2_step(const pevsl_devcsr *B, const double *d, double *x, double *r, double *dnew,
                   double c1, double c2, double *tmp);
/* Same recurrence when A x is computed by a user callback: ax = A vk. */
int cheb_combine(long n, const double *ax, const double *vk, const double *vkm1, double *vkp1,
                 double *y, double cc, double t, double mu0, double muk, int first);
/* KPM: one degree for s <= 64 vectors, row-interleaved with ld = s rounded
 * up to even, Xkp1 = (A Xk - ctr Xk) sc - Xkm1 (Xkm1 may be NULL, and Xkp1
 * may be Xkm1), and per
 * block the sums of <x_{k+1}, x_{k+1}> and <x_{k+1}, x_k> of every column
 * into part (kpm_blocks x 2 ld doubles).  kpm_reduce adds them over the
 * blocks for all steps: out[step][c][0..1] and [2..3], high and low part of
 * each (4 ld doubles per step). */
int kpm_blocks(const pevsl_devcsr *A, int s);
int kpm_step(const pevsl_devcsr *A, int s, const double *Xk, const double *Xkm1, double *Xkp1,
             double ctr, double sc, double *part);
/* the same sums part for <x_0, x_0> of the start vectors (and 0) */
int kpm_start(const pevsl_devcsr *A, int s, const double *X, double *part);
int kpm_reduce(const pevsl_devcsr *A, int s, int steps, const double *part, double *out);
/* vectors that share a group (at most 64) */
int kpm_group(const pevsl_devcsr *A, int nvec);
/* out[c] = sum_b partials[b*s + c] over nb blocks, fixed order */
int col_reduce(const double *partials, int nb, int s, double *out);
/* Column sums of squares of an interleaved block: out[c] = sum_i X[i*ld+c]^2 */
int block_colnorm2(long n, int s, int ld, const double *X, double *out);
/* X[i*ld+c] *= 1/sqrt(nrm2[c]) */
int block_normalize(long n, int s, int ld, double *X, const double *nrm2);

/* ---------------------------------------------------------------- dense */
/* w[j] = sum_i V[i + j*ldv] v[i], j < k (two-stage, deterministic); kernels
 * return early when skip != NULL and *skip == 0 */
int gemvT(long n, int k, const double *V, long ldv, const double *v, double *w, const int *run);
/* v -= V w; *nrm = ||v||; if flag: *flag = (*nrm <= eta * *nrm_old), then
 * *nrm_old = *nrm.  Skipped when run != NULL and *run == 0. */
int gemv_sub_nrm(long n, int k, const double *V, long ldv, const double *w, double *v,
                 double *nrm, const int *run, int *flag_out, double *nrm_old, double eta);
/* ---------------------------------------------------------------- batched
 * Entry s of every call uses pointer p[s] / scalar v[s] and length
 * len.n[s] (leading dimension len.ld[s] for basis blocks); only entries
 * whose bit is set in mask run.  Per-entry outputs go to out[s]. */
struct BLen {
  long n[kMaxBatch];
  long ld[kMaxBatch];
};
BLen blen_uniform(long n, long ld, int S);
int b_axpy(const BLen &len, int S, CPtrs x, VPtrs y, BScal a, unsigned mask);
int b_scal(const BLen &len, int S, VPtrs x, BScal a, unsigned mask);
/* y_s += sign coef[s] x_s, then out[s] = <z_s, y_s>, for all S entries; the
 * scalars in device memory */
int b_axpy_dev_dot(const BLen &len, int S, const double *coef, double sign, CPtrs x, VPtrs y,
                   CPtrs z, double *out);
/* x_s *= 1 / nrm[s] for all S entries, nrm in device memory */
int b_scal_inv_dev(const BLen &len, int S, const double *nrm, VPtrs x);
int b_dot(const BLen &len, int S, CPtrs x, CPtrs y, double *out, int fin, unsigned mask);
int b_axpy_dev_nrm2(const BLen &len, int S, const double *coef, CPtrs x, VPtrs y, double *nrm,
                    unsigned mask);
/* w[s*ldw + j] = <V_s(:,j), v_s>, j < k */
int b_gemvT(const BLen &len, int S, int k, CPtrs V, CPtrs v, double *w, long ldw, const int *run,
            unsigned mask);
/* v_s -= V_s w_s; nrm[s] = ||v_s||; flag/nrm_old per entry as gemv_sub_nrm */
int b_gemv_sub_nrm(const BLen &len, int S, int k, CPtrs V, const double *w, long ldw, VPtrs v,
                   double *nrm, const int *run, int *flag_out, double *nrm_old, double eta,
                   unsigned mask);
/* one filter degree (SRC/chebpol.c:538-568) for nb <= kMaxEntries
 * independent vectors, each on its own matrix A (entries on one matrix read
 * it once per launch): entry e's pointers are FP64 vectors, or FP32 ones
 * when fp32 (then the last degree sets yout, the FP64 result) */
struct ChebEntry {
  const pevsl_devcsr *A;
  const void *vk, *vkm1; /* vkm1 NULL at the first degree */
  void *vkp1, *y;        /* vkp1 may alias vkm1 */
  double *yout;
  double cc, t, mu0, muk;
  int first;
};
int cheb_step_batch(int nb, const ChebEntry *e, bool fp32);
/* the same degree for S in {2,4,8,16} vectors of one problem held
 * row-interleaved (X[i*S + s]); mu0[s], muk[s] on the device; Xkp1 may
 * alias Xkm1 */
int cheb_step_il(const pevsl_devcsr *A, int S, const double *Xk, const double *Xkm1, double *Xkp1,
                 double *Y, double cc, double t, const double *mu0, const double *muk, int first);
/* the same with the SpMV reading Xg instead of Xk (generalized filter) */
int cheb_step_il_x(const pevsl_devcsr *A, int S, const double *Xg, const double *Xk,
                   const double *Xkm1, double *Xkp1, double *Y, double cc, double t,
                   const double *mu0, const double *muk, int first);
/* degree k with a deferred accumulator: Y takes the terms of degrees
 * k-ny+1 .. k (ny in 0..3; 0 leaves Y untouched, neither read nor
 * written), whose vectors are X_k (Xkp1), X_{k-1} (Xk) and X_{k-2} (Xkm1);
 * their mu rows lie at muk, muk - S, muk - 2S.  fresh: Y holds nothing yet
 * and the sum starts from mu_0 X_0 (X_0 = Xk when ny = 1, Xkm1 when
 * ny = 2).  The multiply-adds run in degree order, so Y ends bit-identical
 * to the one-degree-at-a-time sum. */
int cheb_step_il_y(const pevsl_devcsr *A, int S, const double *Xg, const double *Xk,
                   const double *Xkm1, double *Xkp1, double *Y, double cc, double t,
                   const double *mu0, const double *muk, int ny, int fresh);
/* X[i*S + s] = xs[s][i] (S <= kMaxBatch), and ys[s][i] = X[i*S + s] for
 * the first cols columns */
int il_pack(long n, int S, const double *const *xs, double *X);
int il_unpack(long n, int S, int cols, const double *X, double *const *ys);
/* bytes a pass over A reads for the matrix: a row's mask in the stencil
 * form, else per entry 3 (packed: int16 column offset + uint8 value index), 12
 * (int32 column + FP64 value) or 8 (FP32 value), and the row pointers */
double matrix_bytes(const pevsl_devcsr *A, bool fp32, bool batch = false);
/* the same of the interleaved kernels */
double il_matrix_bytes(const pevsl_devcsr *A);
/* L2 persistence window over the part of A the kernels read (if enabled) */
void matrix_window(const pevsl_devcsr *A);
/* choose the CSR-stream form of a matrix by timing (once) */
int stream_tune(pevsl_devcsr *A);
/* choose the CSR or ELL form of the one- and two-vector filter degrees of a
 * packed matrix with an ELL copy by timing both (at set-up) */
int filter_tune(pevsl_devcsr *A);

/* One entry of the persistent filter: y = p(A) x for its own matrix and
 * polynomial (mu on the device).  FP64 entries: b0, b1 are two work vectors
 * of n doubles and acc == y.  FP32 entries (a = the FP32 values): x is the
 * FP32 copy of the input, b0, b1, acc are FP32 and the last degree writes
 * y in FP64. */
struct FiltDev {
  const int *ia, *ja;
  const void *a;
  int n, deg, fp32, pad;
  double cc, t1, t2;
  const double *mu;
  const void *x;
  void *b0, *b1, *acc;
  double *y;
};
constexpr size_t kFiltTabBytes = sizeof(FiltDev) * kMaxEntries + sizeof(int) * (kMaxEntries + 8);
constexpr int kTabSlots = 4; /* staging slots: a slot is reused only after its copy ran */
/* All degrees of ne <= kMaxEntries filters in one cooperative launch: the
 * blocks sweep the (entry, 256-row block) items of every entry whose degree
 * has not been reached, then meet at a grid barrier before the next degree.
 * The entries must be sorted by non-increasing degree.  Returns 0,
 * PEVSL_ERR_CUDA, or PEVSL_ERR_ARG if the launch cannot be co-resident. */
int cheb_filter_persistent(int ne, const FiltDev *entries, int maxdeg);
/* the barrier's timeout flag of the last persistent filter (read after a sync) */
int persistent_filter_error();
void set_barrier_spins(unsigned spins);
int seed_barrier_arrivals(unsigned count);

/* One filter application y = p(A) x of a small problem by one thread-block
 * cluster, all degrees in one launch (gpu_cluster.cu).  With B set each
 * degree is preceded by the B-solve sum_j lmu[j] T_j((B - ccB)/ddB), j <=
 * degB.  mu, lmu: device; deg, degB >= 1; y may alias x. */
struct ClusterJob {
  const pevsl_devcsr *A, *B;
  const double *x;
  double *y;
  const double *mu, *lmu;
  double cc, dd, ccB, ddB;
  int deg, degB;
};
/* largest matrix of a cluster launch */
constexpr int kClusterMaxRows = 32768;
/* A cluster launch costs about 10 us more than the first of the launches per
 * degree (it loads the entries and meets its neighbours twice first) and gains 1
 * to 1.3 us per degree: one vector, 7980 rows, launches / cluster, degree 2 12.4
 * / 20.3 us, 6 20.9 / 23.2, 8 24.8 / 24.5, 24 56.5 / 37.7; 15600 rows 8 25.4 /
 * 28.3, 12 33.5 / 32.5; 6007 rows of 11 scattered entries 8 32.5 / 34.4, 12 45.2
 * / 41.3.  So single applications of lower degree are launched per degree. */
constexpr int kClusterMinDeg = 8;
/* whether the matrices fit the shared memory of a cluster */
bool cluster_filter_ok(const pevsl_devcsr *A, const pevsl_devcsr *B, bool fp32);
/* the applications of ne jobs, all with B or all without */
int cluster_filter(int ne, const ClusterJob *jobs, bool fp32);
/* microseconds after which a block of a cluster launch stops waiting for its
 * neighbours and the call fails; < 0 the default */
void set_cluster_wait(long us);
/* for tests: every block waits for eight bytes that nobody sends */
void withhold_cluster_values(bool on);

/* ---------------------------------------------------------------- FP32 (mixed) */
int csr_make_fp32(pevsl_devcsr *A); /* FP32 copy of the values, once */
int kpm_step32(const pevsl_devcsr *A, int s, int ld, const float *Xk, const float *Xkm1,
               float *Xkp1, const float *V0, double ctr, double sc, double *mom);
int cvt_f64_f32(long n, const double *x, float *y);

/* C = V(:, 0:k)' W(:, 0:m)  (k x m, column-major ldc); deterministic */
int gemm_tn(long n, int k, int m, const double *V, long ldv, const double *W, long ldw, double *C,
            long ldc);
/* the ends of the spectrum of a symmetric n x n host matrix (column major):
 * val[0..3] = lam_1, lam_2, lam_{n-1}, lam_n, val[4..5] the last elements of
 * the eigenvectors of lam_1 and lam_n, which go to Y (device, 2n); waits.
 * ritz_ends_ok: the n it takes */
bool ritz_ends_ok(int n);
int ritz_ends(int n, const double *T, int ldt, double *Y, double *val);
/* U = V(:, 0:k) Y  (n x m, V column-major ldv, Y k x m column-major ldy) */
int gemm_nn(long n, int k, int m, const double *V, long ldv, const double *Y, long ldy,
            double *U, long ldu);

}  // namespace pv

#endif
