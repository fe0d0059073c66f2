/*
 * The solvers of the slicing path, driven from the host with every vector
 * operation on the GPU:
 *
 *   filter application   pEVSL_ChebAv     SRC/chebpol.c:509-574
 *   KPM DOS              pEVSL_Kpmdos     SRC/kpmdos.c:36-197
 *   Lanczos DOS          pEVSL_LanDosG    SRC/landos.c:40-314
 *   spectrum bounds      pEVSL_LanTrbounds SRC/lantrbnd.c:31-408
 *   filtered Lanczos     pEVSL_ChebLanNr  SRC/cheblanNr.c:54-448
 *
 * The control flow (step counts, tests, breakdown restarts, acceptance) is
 * the reference's.  ChebLanNr's host side reads two scalars per Lanczos step
 * (alpha, beta), the bounds' and the Lanczos DOS's those of a whole cycle or
 * run at once (lan_step); everything else stays on the device.  The DGKS second
 * Gram-Schmidt pass is decided on the device.  When A is the built-in
 * parcsr, the SpMV is fused into the recurrence kernels; a user matvec
 * (pEVSL_SetAMatvec) is called with device pointers instead.
 */
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <thread>
#include <vector>

#include "gpu.cuh"
#include "gpu_device.cuh"

using namespace pv;

namespace {

const double kEta = 0.70710678118654752440; /* 1/sqrt(2): DGKS threshold */

/* ------------------------------------------------------------ event timer
 * Sums the device time of repeated segments (filter applications,
 * reorthogonalisation) with a small pool of event pairs that is drained
 * whenever it fills; the pools live for the whole process. */
struct SegTimer {
  static constexpr int kPairs = 64;
  cudaEvent_t ev[2 * kPairs];
  int used = 0;
  double acc_ms = 0.0;
  bool ok = false;
  void init() {
    if (!ok) {
      ok = true;
      for (int i = 0; i < 2 * kPairs; i++)
        if (cudaEventCreate(&ev[i]) != cudaSuccess) ok = false;
    }
    used = 0;
    acc_ms = 0.0;
  }
  void begin() {
    if (!ok) return;
    if (used == kPairs) flush();
    cudaEventRecord(ev[2 * used], ctx().stream);
  }
  void end() {
    if (!ok) return;
    cudaEventRecord(ev[2 * used + 1], ctx().stream);
    used++;
  }
  void flush() {
    if (!ok || used == 0) return;
    cudaEventSynchronize(ev[2 * used - 1]);
    for (int i = 0; i < used; i++) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]) == cudaSuccess) acc_ms += ms;
    }
    used = 0;
  }
};
SegTimer g_t_pol, g_t_orth;

/* process-wide counters of the fused filter kernel (pEVSL_B200_FilterCounters) */
uint64_t g_filter_launches = 0;
uint64_t g_filter_persistent = 0; /* persistent filter launches (each covers many degrees) */
double g_filter_bytes = 0.0;
double g_filter_ms = 0.0;

/* algorithmic HBM bytes of one fused filter degree: the CSR (int32 column
 * indices, fp64 values, int32 row pointers) plus v_k read once, and
 * v_{k-1}, y read / v_{k+1}, y written (first degree: no v_{k-1}, y only
 * written) */
double cheb_step_bytes(const pevsl_devcsr *A, int first) {
  const double n = A->nrows;
  return matrix_bytes(A, false) + (first ? 24.0 : 40.0) * n;
}

/* matvec through the installed operator: fused kernels use the device CSR
 * directly; this is for the plain y = A x steps. */
int apply_A(pevsl_Data *pevsl, const double *x, double *y) {
  pevsl_devcsr *A = pevsl_builtin_A(pevsl);
  pevsl->stats->n_mvA++;
  if (A) return spmv(A, x, y);
  if (!pevsl->Amv || !pevsl->Amv->func) return PEVSL_ERR_NOMATVEC;
  if (sync()) return PEVSL_ERR_CUDA;
  pevsl->Amv->func((double *)x, y, pevsl->Amv->data);
  return fail(cudaDeviceSynchronize(), "user matvec");
}

/* y = p((A - cc)/dd) v with mu[0..deg]; w3 holds 3n doubles; y may be v. */
int cheb_apply(pevsl_Data *pevsl, const pevsl_Polparams *pol, const double *v, double *y,
               double *w3, long n) {
  pevsl_devcsr *A = pevsl_builtin_A(pevsl);
  const int m = pol->deg;
  const double cc = pol->cc, dd = pol->dd;
  const double *mu = pol->mu;
  pevsl->stats->n_polAv++;
  if (m <= 0) {
    if (vcopy(v, y, n)) return PEVSL_ERR_CUDA;
    return vscal(y, n, mu[0]);
  }
  if (!A && (!pevsl->Amv || !pevsl->Amv->func)) return PEVSL_ERR_NOMATVEC;
  if (A && m >= kClusterMinDeg && cluster_filter_ok(A, nullptr, false)) {
    /* a small problem: every degree in one launch, the same bits */
    double *dmu = (double *)ws(WS_CLMU, sizeof(double) * (size_t)(m + 1));
    if (!dmu) return PEVSL_ERR_NOMEM;
    if (memcpy_async(dmu, mu, sizeof(double) * (size_t)(m + 1))) return PEVSL_ERR_CUDA;
    const ClusterJob J{A, nullptr, v, y, dmu, nullptr, cc, dd, 0.0, 0.0, m, 0};
    for (int k = 1; k <= m; k++) g_filter_bytes += cheb_step_bytes(A, k == 1);
    g_filter_launches += (uint64_t)m;
    pevsl->stats->n_mvA += (size_t)m;
    return cluster_filter(1, &J, false);
  }
  double *buf[2] = {w3, w3 + n};
  if (y == v) { /* the first degree's rows read their neighbours' v */
    if (vcopy(v, w3 + 2 * n, n)) return PEVSL_ERR_CUDA;
    v = w3 + 2 * n;
  }
  if (A) {
    g_filter_launches += (uint64_t)m;
    pevsl->stats->n_mvA += (size_t)m;
    return cheb_degrees(A, mu, m, cc, dd, v, y, buf[0], buf[1], &g_filter_bytes);
  }
  double *ax = (double *)ws(WS_VEC, sizeof(double) * (size_t)n);
  if (!ax) return PEVSL_ERR_NOMEM;
  const double *vk = v, *vkm1 = nullptr;
  for (int k = 1; k <= m; k++) {
    double *vkp1 = k <= 2 ? buf[k - 1] : const_cast<double *>(vkm1);
    int st = apply_A(pevsl, vk, ax);
    if (!st)
      st = cheb_combine(n, ax, vk, vkm1, vkp1, y, cc, (k == 1 ? 1.0 : 2.0) / dd, mu[0], mu[k],
                        k == 1);
    pevsl->stats->n_mvA--; /* counted below */
    if (st) return st;
    vkm1 = vk;
    vk = vkp1;
  }
  pevsl->stats->n_mvA += (size_t)m;
  return 0;
}

/* One filter application of a batch: y = p(A) x (pEVSL_ChebAv,
 * SRC/chebpol.c:509-574) for entry e with its own device CSR, polynomial
 * and work space of 16 * ld bytes (two FP64 recurrence vectors, or, in
 * FP32, the FP32 copy of x, two FP32 recurrence vectors and the FP32
 * accumulator; the last degree writes y in FP64). */
struct FilterJob {
  pevsl_Data *pevsl;          /* statistics */
  const pevsl_devcsr *A;
  const double *x;
  double *y;
  const pevsl_Polparams *pol;
  const double *dmu;          /* pol->mu on the device (persistent form) */
  void *work;
  long ld;                    /* spacing of the work vectors: >= n, 256-byte multiple */
};

/* Form of the batched filter: 0 = one cheb_step_batch launch per degree
 * serving every entry (any matrices, up to kMaxEntries), 1 = one persistent
 * cooperative launch for all degrees and entries, 2 (default) = the
 * launches of form 0 captured in a CUDA graph per set of live slices and
 * replayed (filter_graphed).  One launch per degree beat the persistent
 * kernel (81 vs 119 us per degree for 4 slices at 10^6 rows, 4.1 vs 6.1 us
 * at 8000 rows): the grid barrier costs more than the gap between launches. */
static int g_filter_form_override = -1; /* -1: not read yet */
static int filter_form_setting() {
  if (g_filter_form_override < 0) {
    const char *e = getenv("PEVSL_B200_FILTER_FORM");
    const int v = e ? atoi(e) : 2;
    g_filter_form_override = (v >= 0 && v <= 2) ? v : 2;
  }
  return g_filter_form_override;
}
static int filter_form() { return filter_form_setting() == 1 ? 1 : 0; }

/* Interleaved form of the batched filter (PEVSL_B200_INTERLEAVE: 1 on, the
 * default; 0 off): the live slices of one problem on one matrix run with
 * their vectors row-interleaved, so one gather serves every slice
 * (cheb_step_il); the input is packed once and the result unpacked once per
 * filter application.  Applies to 2..16 FP64 slices on a short-row matrix
 * whose polynomials share the spectrum bounds (cc, dd) (il_partition).  Measured per
 * degree against the grid-interleaved batch kernel: 100^3, 4 slices 52.6
 * vs 80.1 us (2 slices 34.0 vs 44.6, 16 slices 182 vs 310); random sparse
 * n = 2e6 with ~17 entries per row, 16 slices 758 vs 2160 us. */
static int interleave_setting() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("PEVSL_B200_INTERLEAVE");
    v = e ? atoi(e) != 0 : 1;
  }
  return v;
}

static int il_width(int nlive) { return nlive <= 2 ? 2 : nlive <= 4 ? 4 : nlive <= 8 ? 8 : 16; }

/* Slices per interleaved group.  A group runs all its degrees, and its
 * working set from one degree to the next -- three row-interleaved vector
 * blocks (24 n bytes per slice) and the matrix -- stays in the 126 MB L2 when
 * it is at most half of it; wider groups stream it from HBM at every degree.
 * So a group holds the most slices (2, 4, 8 or 16) that fit in 64 MB (stencil
 * matrices, whose mask is nearly nothing: 70), at least 2.  Stencil matrices
 * per degree, four slices as one group / as two: 80 x 81 x 79 (48 MB) 8.4 /
 * 10.2 us, 90 x 91 x 89 (70 MB) 12.0 / 13.3, 99 x 100 x 101 (96 MB) 19.0 /
 * 17.0; eight as one / as two of four: 72 x 71 x 73 (72 MB) 11.9 / 13.4, 80 x
 * 81 x 79 (97 MB) 18.8 / 16.8.  PEVSL_B200_IL_MAXS caps it by hand (2..16). */
static int il_group_cap(const pevsl_devcsr *A) {
  const char *e = getenv("PEVSL_B200_IL_MAXS"); /* read per call: tests change it */
  const int env = e ? atoi(e) : 0;
  if (env >= 2) return PEVSL_MIN(env, kMaxBatch);
  const double mat = A->smask ? il_matrix_bytes(A) : 3.0 * (double)A->nnz + 4.0 * (A->nrows + 1.0);
  const double most = (A->smask ? 70.0 : 64.0) * 1024 * 1024;
  int cap = 2;
  for (int S = 4; S <= kMaxBatch; S *= 2)
    if (24.0 * (double)A->nrows * S + mat <= most) cap = S;
  return cap;
}

/* Degrees per accumulator update in the interleaved filter
 * (PEVSL_B200_IL_DEFER: 1, 2 or 3, the default).  With D > 1 a launch adds
 * the terms of the last D degrees to y (the first update at degree
 * min(D, 2), the last at the group's top degree) and the launches between
 * updates neither read nor write y: 24 instead of 40 bytes per row and
 * slice.  The sum is the same, term by term in degree order. */
static int il_defer_setting() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("PEVSL_B200_IL_DEFER");
    v = e ? atoi(e) : 3;
    if (v < 1 || v > 3) v = 3;
  }
  return v;
}

static constexpr double kBranchBytes = 64.0 * 1024 * 1024;

/* a set of slices the interleaved form serves together */
struct IlGroup {
  const pevsl_devcsr *A;
  int idx[kMaxBatch]; /* job indices, in job order */
  int cnt, S, maxdeg;
  double cc, dd;
  size_t ws_off, mu_off; /* in doubles, into WS_IL / WS_ILMU */
};

/* The entries the interleaved form takes: groups of 2..16 live FP64
 * entries on one short-row matrix with the same spectrum bounds (cc, dd), in
 * job order, that is in the stencil form or has at least 2^16 rows, and is
 * too large for a cluster; the other entries stay with the grid-interleaved
 * batch kernel.  Below 2^16 rows the plain kernel is latency-bound, where
 * the batch kernel is faster (20^3, 5 slices: the whole run 0.115 vs 0.125
 * s). */
static void il_partition(int ne, const FilterJob *jobs, bool fp32, std::vector<IlGroup> &g,
                         std::vector<char> &taken) {
  g.clear();
  taken.assign((size_t)ne, 0);
  if (fp32 || !interleave_setting()) return;
  std::vector<char> seen((size_t)ne, 0);
  size_t ws_off = 0, mu_off = 0;
  for (int e = 0; e < ne; e++) {
    const FilterJob &J = jobs[e];
    if (seen[e] || J.pol->deg <= 0) continue;
    const pevsl_devcsr *A = J.A;
    if (A->lanes != 0 || (A->nrows < 65536 && !A->smask) || cluster_filter_ok(A, nullptr, false))
      continue;
    std::vector<int> L;
    for (int f = e; f < ne; f++)
      if (!seen[f] && jobs[f].pol->deg > 0 && jobs[f].A == A && jobs[f].pol->cc == J.pol->cc &&
          jobs[f].pol->dd == J.pol->dd) {
        seen[f] = 1;
        L.push_back(f);
      }
    const size_t cap = (size_t)il_group_cap(A);
    for (size_t c0 = 0; c0 < L.size(); c0 += cap) {
      const int cnt = (int)PEVSL_MIN(cap, L.size() - c0);
      if (cnt < 2) continue;
      IlGroup G;
      G.A = A;
      G.cnt = cnt;
      G.S = il_width(cnt);
      G.maxdeg = 0;
      G.cc = J.pol->cc;
      G.dd = J.pol->dd;
      for (int i = 0; i < cnt; i++) {
        G.idx[i] = L[c0 + i];
        taken[(size_t)G.idx[i]] = 1;
        G.maxdeg = PEVSL_MAX(G.maxdeg, jobs[G.idx[i]].pol->deg);
      }
      G.ws_off = ws_off;
      G.mu_off = mu_off;
      ws_off += 4 * (size_t)A->nrows * (size_t)G.S;
      mu_off += (size_t)(G.maxdeg + 1) * (size_t)G.S;
      g.push_back(G);
    }
  }
}

static size_t il_ws_doubles(const std::vector<IlGroup> &g) {
  return g.empty() ? 0 : g.back().ws_off + 4 * (size_t)g.back().A->nrows * (size_t)g.back().S;
}
static size_t il_mu_doubles(const std::vector<IlGroup> &g) {
  return g.empty() ? 0 : g.back().mu_off + (size_t)(g.back().maxdeg + 1) * (size_t)g.back().S;
}

/* workspace and per-degree coefficient tables of the interleaved groups,
 * prepared outside any stream capture: row k of a group's table holds mu_k
 * of each of its slices (0 past a slice's degree, where its y then stays
 * unchanged) */
static int il_prepare(int ne, const FilterJob *jobs, bool fp32) {
  std::vector<IlGroup> g;
  std::vector<char> taken;
  il_partition(ne, jobs, fp32, g, taken);
  if (g.empty()) return 0;
  if (!ws(WS_IL, sizeof(double) * il_ws_doubles(g))) return PEVSL_ERR_NOMEM;
  double *dmu = (double *)ws(WS_ILMU, sizeof(double) * il_mu_doubles(g));
  if (!dmu) return PEVSL_ERR_NOMEM;
  std::vector<double> tab(il_mu_doubles(g), 0.0);
  for (const IlGroup &G : g)
    for (int c = 0; c < G.cnt; c++) {
      const pevsl_Polparams *pol = jobs[G.idx[c]].pol;
      for (int k = 0; k <= pol->deg; k++) tab[G.mu_off + (size_t)k * G.S + c] = pol->mu[k];
    }
  if (memcpy_async(dmu, tab.data(), sizeof(double) * tab.size())) return PEVSL_ERR_CUDA;
  return sync();
}

/* buffers of group G: packed input, two recurrence blocks, accumulator */
static void il_buffers(const IlGroup &G, double **X0, double **B0, double **B1, double **Y) {
  const size_t blk = (size_t)G.A->nrows * (size_t)G.S;
  *X0 = (double *)ctx().ws[WS_IL] + G.ws_off;
  *B0 = *X0 + blk;
  *B1 = *B0 + blk;
  *Y = *B1 + blk;
}

static double filter_bytes_degree(const pevsl_devcsr *A, int deg_k, bool fp32, bool last) {
  const double n = A->nrows, vb = fp32 ? 4.0 : 8.0;
  return (deg_k == 1 ? 3.0 : 5.0) * vb * n + (last ? 4.0 * n : 0.0);
}

/* the group's inputs from the jobs' x, and its results to their y */
static int il_pack_group(const IlGroup &G, const FilterJob *jobs) {
  const double *xs[kMaxBatch];
  for (int c = 0; c < G.S; c++) xs[c] = jobs[G.idx[c < G.cnt ? c : 0]].x; /* padding: mu 0 */
  double *X0, *B0, *B1, *Y;
  il_buffers(G, &X0, &B0, &B1, &Y);
  return il_pack(G.A->nrows, G.S, xs, X0);
}
static int il_unpack_group(const IlGroup &G, const FilterJob *jobs) {
  double *ys[kMaxBatch];
  for (int c = 0; c < G.cnt; c++) ys[c] = jobs[G.idx[c]].y;
  double *X0, *B0, *B1, *Y;
  il_buffers(G, &X0, &B0, &B1, &Y);
  return il_unpack(G.A->nrows, G.S, G.cnt, Y, ys);
}

/* Branches of a captured application: the groups over up to kSideStreams + 1
 * branches, the longest first to the branch with the least time.  A group
 * alone is bound by the latency of its degrees, so several at a time gain as
 * long as they stay in L2 together: the largest working sets of the branches
 * must sum to at most kBranchBytes, else there is one branch less.  Returns
 * their number.  Whole runs, one after another / as branches: three grids of
 * 216000, 32399 and 21924 rows with three slices each 391 / 275 ms, two of
 * 216000 with three 513 / 372, four of 85000 with three 415 / 242, 40 slices
 * at 26970 rows (three groups) 864 / 550; with a limit of 110 MB two groups of
 * two at 10^6 rows 2.51 -> 2.71 s.  (The cluster launch of small problems
 * stays ahead of them: beside the groups its blocks and theirs share SMs, and
 * 7980 rows with 216000 gained 4%.) */
static int filter_branches(const std::vector<IlGroup> &g, std::vector<int> *branch) {
  const size_t ng = g.size();
  std::vector<double> us(ng), bytes(ng);
  std::vector<size_t> ord(ng);
  for (size_t i = 0; i < ng; i++) {
    const double v = 24.0 * (double)g[i].A->nrows * g[i].S;
    ord[i] = i;
    bytes[i] = v + il_matrix_bytes(g[i].A);
    us[i] = g[i].maxdeg * (1.5 + v / 5e6); /* latency, and 5 TB/s */
  }
  std::sort(ord.begin(), ord.end(), [&](size_t a, size_t b) { return us[a] > us[b]; });
  for (int nb = (int)PEVSL_MIN((size_t)kSideStreams + 1, ng); nb > 1; nb--) {
    std::vector<double> load((size_t)nb, 0.0), most((size_t)nb, 0.0);
    for (size_t i : ord) {
      const size_t b = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
      (*branch)[i] = (int)b;
      load[b] += us[i];
      most[b] = PEVSL_MAX(most[b], bytes[i]);
    }
    double sum = 0.0;
    for (double m : most) sum += m;
    if (sum <= kBranchBytes) return nb;
  }
  std::fill(branch->begin(), branch->end(), 0);
  return 1;
}

/* The side streams only ever carry work inside a capture of the context
 * stream, as branches of its graph: what runs, runs in the graph's launch on
 * the context stream. */
static int fork_branches(int nb) {
  Ctx &c = ctx();
  if (fail(cudaEventRecord(c.side_ev[0], c.stream), "cudaEventRecord")) return PEVSL_ERR_CUDA;
  for (int b = 1; b < nb; b++)
    if (fail(cudaStreamWaitEvent(c.side[b - 1], c.side_ev[0], 0), "cudaStreamWaitEvent"))
      return PEVSL_ERR_CUDA;
  return 0;
}
static int join_branches(int nb) {
  Ctx &c = ctx();
  int st = 0;
  for (int b = 1; b < nb; b++)
    if (fail(cudaEventRecord(c.side_ev[b], c.side[b - 1]), "cudaEventRecord") ||
        fail(cudaStreamWaitEvent(c.stream, c.side_ev[b], 0), "cudaStreamWaitEvent"))
      st = PEVSL_ERR_CUDA;
  return st;
}
/* launches go to branch b's stream while one of these is alive */
struct BranchScope {
  cudaStream_t main;
  explicit BranchScope(int b) : main(ctx().stream) {
    if (b > 0) ctx().stream = ctx().side[b - 1];
  }
  ~BranchScope() { ctx().stream = main; }
};
static int branch_streams() {
  Ctx &c = ctx();
  for (int b = 0; b <= kSideStreams; b++) {
    if (!c.side_ev[b] &&
        fail(cudaEventCreateWithFlags(&c.side_ev[b], cudaEventDisableTiming), "cudaEventCreate"))
      return PEVSL_ERR_CUDA;
    if (b < kSideStreams && !c.side[b] &&
        fail(cudaStreamCreateWithFlags(&c.side[b], cudaStreamNonBlocking), "cudaStreamCreate"))
      return PEVSL_ERR_CUDA;
  }
  return 0;
}

/* packed: the interleaved groups' inputs are in their buffers and the results
 * stay there */
static int cheb_filter_batch(int ne, const FilterJob *jobs, bool fp32, bool packed = false) {
  if (ne <= 0) return 0;
  if (ne > kMaxEntries) return PEVSL_ERR_ARG;
  int st = 0, maxdeg = 0, nlive = 0;
  int live[kMaxEntries];
  for (int e = 0; e < ne && !st; e++) {
    const FilterJob &J = jobs[e];
    const pevsl_Polparams *pol = J.pol;
    const long n = J.A->nrows;
    if (fp32 && !J.A->a32) return PEVSL_ERR_ARG;
    J.pevsl->stats->n_polAv++;
    J.pevsl->stats->n_mvA += (size_t)PEVSL_MAX(pol->deg, 0);
    if (pol->deg <= 0) {
      st = vcopy(J.x, J.y, n);
      if (!st) st = vscal(J.y, n, pol->mu[0]);
      continue;
    }
    maxdeg = PEVSL_MAX(maxdeg, pol->deg);
    /* the cluster form converts its input itself */
    if (fp32 && (filter_form() == 1 || !cluster_filter_ok(J.A, nullptr, true)))
      st = cvt_f64_f32(n, J.x, (float *)J.work);
    live[nlive++] = e;
  }
  if (st || !nlive) return st;
  /* matrix bytes: each distinct matrix once per degree, up to the largest
   * degree of its entries */
  double mat_bytes = 0.0;
  for (int i = 0; i < nlive; i++) {
    const pevsl_devcsr *A = jobs[live[i]].A;
    bool seen = false;
    for (int t = 0; t < i && !seen; t++) seen = jobs[live[t]].A == A;
    if (seen) continue;
    int dmax = 0;
    for (int t = i; t < nlive; t++)
      if (jobs[live[t]].A == A) dmax = PEVSL_MAX(dmax, jobs[live[t]].pol->deg);
    mat_bytes += (double)dmax * ((fp32 ? 8.0 : 12.0) * (double)A->nnz + 4.0 * (A->nrows + 1.0));
  }
  const int form = filter_form();
  if (form == 1) {
    /* table sorted by non-increasing degree (stable: ties keep their order) */
    FiltDev tab[kMaxEntries];
    int ord[kMaxEntries];
    for (int i = 0; i < nlive; i++) ord[i] = live[i];
    for (int i = 1; i < nlive; i++) {
      const int v = ord[i];
      int j = i - 1;
      while (j >= 0 && jobs[ord[j]].pol->deg < jobs[v].pol->deg) {
        ord[j + 1] = ord[j];
        j--;
      }
      ord[j + 1] = v;
    }
    double bytes = mat_bytes;
    for (int i = 0; i < nlive; i++) {
      const FilterJob &J = jobs[ord[i]];
      const pevsl_devcsr *A = J.A;
      FiltDev &E = tab[i];
      E.ia = A->ia;
      E.ja = A->ja;
      E.a = fp32 ? (const void *)A->a32 : (const void *)A->a;
      E.n = (int)A->nrows;
      E.deg = J.pol->deg;
      E.fp32 = fp32;
      E.pad = 0;
      E.cc = J.pol->cc;
      E.t1 = 1.0 / J.pol->dd;
      E.t2 = 2.0 / J.pol->dd;
      E.mu = J.dmu;
      if (fp32) {
        float *w = (float *)J.work;
        E.x = w;
        E.b0 = w + J.ld;
        E.b1 = w + 2 * J.ld;
        E.acc = w + 3 * J.ld;
      } else {
        double *w = (double *)J.work;
        E.x = J.x;
        E.b0 = w;
        E.b1 = w + J.ld;
        E.acc = J.y;
      }
      E.y = J.y;
      for (int k = 1; k <= E.deg; k++) bytes += filter_bytes_degree(A, k, fp32, fp32 && k == E.deg);
    }
    st = cheb_filter_persistent(nlive, tab, maxdeg);
    g_filter_launches += (uint64_t)maxdeg;
    g_filter_bytes += bytes;
    g_filter_persistent++;
    /* a barrier wait that ran out leaves the filter half applied: report it
     * before anything uses the result (one 16-byte read per application) */
    if (!st && persistent_filter_error()) {
      fprintf(stderr, "pevsl_b200: persistent filter barrier timed out\n");
      st = PEVSL_ERR_CUDA;
    }
    return st;
  }
  /* one launch per degree for all live entries; a matrix is read once per
   * launch for all entries on it.  Entries taken by interleaved groups run
   * as one interleaved launch per group and degree instead, small problems
   * as one cluster launch for all their degrees. */
  std::vector<IlGroup> ig;
  std::vector<char> taken;
  il_partition(ne, jobs, fp32, ig, taken);
  std::vector<ClusterJob> cj;
  for (int i = 0; i < nlive; i++) {
    const FilterJob &J = jobs[live[i]];
    if (taken[(size_t)live[i]] || !cluster_filter_ok(J.A, nullptr, fp32)) continue;
    taken[(size_t)live[i]] = 1;
    cj.push_back(ClusterJob{J.A, nullptr, J.x, J.y, J.dmu, nullptr, J.pol->cc, J.pol->dd, 0.0, 0.0,
                            J.pol->deg, 0});
  }
  const int defer = il_defer_setting();
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(ctx().stream, &cs);
  const bool capturing = cs != cudaStreamCaptureStatusNone;
  if (!ig.empty()) {
    /* inside a capture the caller prepared the workspace and coefficients */
    if (!capturing) st = il_prepare(ne, jobs, fp32);
    if (!st && (!ctx().ws[WS_IL] || ctx().wsz[WS_IL] < sizeof(double) * il_ws_doubles(ig) ||
                !ctx().ws[WS_ILMU] || ctx().wsz[WS_ILMU] < sizeof(double) * il_mu_doubles(ig)))
      st = PEVSL_ERR_ARG; /* il_prepare not run before the capture */
    if (st) return st;
  }
  auto clusters = [&]() -> int {
    if (cj.empty()) return 0;
    const int r = cluster_filter((int)cj.size(), cj.data(), fp32);
    if (r) return r;
    int dmax = 0;
    for (size_t i = 0; i < cj.size(); i++) {
      const pevsl_devcsr *A = cj[i].A;
      dmax = PEVSL_MAX(dmax, cj[i].deg);
      for (int k = 1; k <= cj[i].deg; k++)
        g_filter_bytes += filter_bytes_degree(A, k, fp32, fp32 && k == cj[i].deg) +
                          matrix_bytes(A, fp32);
    }
    g_filter_launches += (uint64_t)dmax;
    return 0;
  };
  /* a group through all its degrees, so that its working set stays in L2
   * between them (il_group_cap); the groups are independent, so every
   * slice's bits are those of the degree-major order */
  auto group = [&](const IlGroup &G) -> int {
    int r = packed ? 0 : il_pack_group(G, jobs);
    double *X0, *B0, *B1, *Y;
    il_buffers(G, &X0, &B0, &B1, &Y);
    const double *dmu = (const double *)ctx().ws[WS_ILMU] + G.mu_off;
    const double *gk = X0, *gkm1 = nullptr;
    for (int k = 1, lastw = 0; k <= G.maxdeg && !r; k++) {
      double *gkp1 = k == 1 ? B0 : k == 2 ? B1 : const_cast<double *>(gkm1);
      const int ny = deferred_terms(k, lastw, G.maxdeg, defer), fresh = ny > 0 && lastw == 0;
      r = cheb_step_il_y(G.A, G.S, gk, gk, gkm1, gkp1, Y, G.cc, (k == 1 ? 1.0 : 2.0) / G.dd, dmu,
                         dmu + (size_t)k * G.S, ny, fresh);
      if (ny > 0) lastw = k;
      /* read v_k, v_{k-1} (from degree 2), write v_{k+1}; y read unless
       * fresh and written when updated */
      const double vec = (k == 1 ? 16.0 : 24.0) + (ny > 0 ? (fresh ? 8.0 : 16.0) : 0.0);
      g_filter_bytes += il_matrix_bytes(G.A) + vec * (double)G.A->nrows * G.S;
      g_filter_launches++;
      gkm1 = gk;
      gk = gkp1;
    }
    if (!r && !packed) r = il_unpack_group(G, jobs);
    return r;
  };
  st = clusters();
  if (st) return st;
  /* in a capture the groups become parallel branches of the graph */
  std::vector<int> branch(ig.size(), 0);
  const int nb = capturing ? filter_branches(ig, &branch) : 1;
  if (nb > 1 && (st = fork_branches(nb))) return st;
  for (int b = nb - 1; b >= 0 && !st; b--) {
    BranchScope on(b);
    for (size_t gi = 0; gi < ig.size() && !st; gi++)
      if (branch[gi] == b) st = group(ig[gi]);
  }
  std::vector<const void *> vk(nlive), vkm1(nlive);
  std::vector<void *> b0(nlive), b1(nlive), acc(nlive);
  for (int i = 0; i < nlive; i++) {
    const FilterJob &J = jobs[live[i]];
    if (fp32) {
      float *w = (float *)J.work;
      vk[i] = w;
      b0[i] = w + J.ld;
      b1[i] = w + 2 * J.ld;
      acc[i] = w + 3 * J.ld;
    } else {
      double *w = (double *)J.work;
      vk[i] = J.x;
      b0[i] = w;
      b1[i] = w + J.ld;
      acc[i] = J.y;
    }
    vkm1[i] = nullptr;
  }
  int nother = 0, other = -1;
  maxdeg = 0;
  for (int i = 0; i < nlive; i++)
    if (!taken[(size_t)live[i]]) {
      nother++;
      other = i;
      maxdeg = PEVSL_MAX(maxdeg, jobs[live[i]].pol->deg);
    }
  bool others = nother > 0;
  if (!st && nother == 1 && !fp32 && jobs[live[other]].A->lanes == 0) {
    /* one slice outside the groups: all its degrees */
    const FilterJob &J = jobs[live[other]];
    st = cheb_degrees(J.A, J.pol->mu, maxdeg, J.pol->cc, J.pol->dd, J.x, J.y, (double *)b0[other],
                      (double *)b1[other], &g_filter_bytes);
    g_filter_launches += (uint64_t)maxdeg;
    others = false;
  }
  std::vector<ChebEntry> en(nlive);
  for (int k = 1; k <= maxdeg && !st && others; k++) {
    int nb = 0;
    double bytes = 0.0;
    for (int i = 0; i < nlive; i++) {
      const FilterJob &J = jobs[live[i]];
      const pevsl_Polparams *pol = J.pol;
      if (taken[(size_t)live[i]]) continue;
      if (k > pol->deg) continue;
      /* two work vectors: from degree 3 on, v_{k+1} replaces v_{k-1} */
      void *vkp1 = k == 1 ? b0[i] : k == 2 ? b1[i] : const_cast<void *>(vkm1[i]);
      const bool last = fp32 && k == pol->deg;
      en[nb++] = ChebEntry{J.A, vk[i], vkm1[i], vkp1, acc[i], last ? J.y : nullptr,
                           pol->cc, (k == 1 ? 1.0 : 2.0) / pol->dd, pol->mu[0], pol->mu[k],
                           k == 1};
      bytes += filter_bytes_degree(J.A, k, fp32, last);
      vkm1[i] = vk[i];
      vk[i] = vkp1;
    }
    /* matrix bytes: each distinct matrix of this degree's entries once */
    for (int i = 0; i < nb; i++) {
      bool seen = false;
      for (int t = 0; t < i && !seen; t++) seen = en[t].A == en[i].A;
      if (!seen)
        bytes += matrix_bytes(en[i].A, fp32, nb > 1);
    }
    if (nb == 0) {
      /* every live entry of this degree is in an interleaved group */
    } else if (nb == 1 && !fp32 && en[0].A->lanes == 0) {
      /* one live slice: the one-vector kernel (packed entries when the
       * matrix has them); the same arithmetic as the batch */
      const ChebEntry &c = en[0];
      st = cheb_step(c.A, (const double *)c.vk, (const double *)c.vkm1, (double *)c.vkp1,
                     (double *)c.y, c.cc, c.t, c.mu0, c.muk, c.first);
    } else {
      st = cheb_step_batch(nb, en.data(), fp32);
    }
    g_filter_launches++;
    g_filter_bytes += bytes;
  }
  if (nb > 1) {
    const int r = join_branches(nb);
    if (!st) st = r;
  }
  return st;
}

/* CUDA graph form of one batched filter application.  The degrees read the
 * input from, and accumulate into, two staging vectors in each slice's
 * work space (at 16 ld and 24 ld bytes), so that the launch sequence of a
 * given set of slices never changes: it is captured once (all degrees, the
 * FP32 conversion included) and replayed, with one copy in and one copy out
 * per slice around it.  A new set of live slices is captured anew. */
static bool filter_graph_enabled() { return filter_form_setting() == 2; }

/* whether every job runs as a cluster launch (or is a copy) */
static bool all_cluster(const std::vector<FilterJob> &jobs, bool fp32) {
  for (const FilterJob &J : jobs)
    if (J.pol->deg > 0 && !cluster_filter_ok(J.A, nullptr, fp32)) return false;
  return true;
}

struct FilterGraph {
  cudaGraphExec_t exec = nullptr;
  std::vector<char> key; /* live slices of the captured sequence */
  std::vector<IlGroup> groups;
  std::vector<char> grouped; /* the jobs in them */
  bool mixed = false;
  uint64_t launches = 0, kernel_launches = 0;
  double bytes = 0.0;
  ~FilterGraph() {
    if (exec) cudaGraphExecDestroy(exec);
  }
};

static int filter_graphed(FilterGraph &fg, const std::vector<char> &sel, std::vector<FilterJob> &jobs) {
  Ctx &c = ctx();
  const int ne = (int)jobs.size();
  std::vector<FilterJob> staged(jobs);
  int st = 0;
  const bool renew = !fg.exec || fg.key != sel;
  if (renew) {
    fg.groups.clear();
    fg.grouped.assign((size_t)ne, 0);
    if (filter_form() == 0) {
      if ((st = il_prepare(ne, jobs.data(), fg.mixed)) || (st = branch_streams())) return st;
      il_partition(ne, jobs.data(), fg.mixed, fg.groups, fg.grouped);
    }
  }
  /* the groups are packed and unpacked around the graph, the others staged */
  for (const IlGroup &G : fg.groups)
    if ((st = il_pack_group(G, jobs.data()))) return st;
  for (int e = 0; e < ne && !st; e++) {
    if (fg.grouped[(size_t)e]) continue;
    double *xs = (double *)((char *)jobs[e].work + 16 * (size_t)jobs[e].ld);
    st = memcpy_async(xs, jobs[e].x, sizeof(double) * (size_t)jobs[e].A->nrows);
    staged[e].x = xs;
    staged[e].y = xs + jobs[e].ld;
  }
  if (st) return st;
  if (renew) {
    if (fg.exec) cudaGraphExecDestroy(fg.exec);
    fg.exec = nullptr;
    const uint64_t l0 = g_filter_launches, k0 = c.launches;
    const double b0 = g_filter_bytes;
    if (fail(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal), "BeginCapture"))
      return PEVSL_ERR_CUDA;
    st = cheb_filter_batch(ne, staged.data(), fg.mixed, true);
    cudaGraph_t gr = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(c.stream, &gr);
    if (st || fail(ec, "EndCapture")) {
      if (gr) cudaGraphDestroy(gr);
      return st ? st : PEVSL_ERR_CUDA;
    }
    const cudaError_t ei = cudaGraphInstantiate(&fg.exec, gr, 0);
    cudaGraphDestroy(gr);
    if (fail(ei, "cudaGraphInstantiate")) {
      fg.exec = nullptr;
      return PEVSL_ERR_CUDA;
    }
    fg.key = sel;
    fg.launches = g_filter_launches - l0;
    fg.kernel_launches = c.launches - k0;
    fg.bytes = g_filter_bytes - b0;
  } else {
    /* the statistics a direct call would have counted */
    for (int e = 0; e < ne; e++) {
      jobs[e].pevsl->stats->n_polAv++;
      jobs[e].pevsl->stats->n_mvA += (size_t)PEVSL_MAX(jobs[e].pol->deg, 0);
    }
    g_filter_launches += fg.launches;
    g_filter_bytes += fg.bytes;
    c.launches += fg.kernel_launches;
  }
  if (fail(cudaGraphLaunch(fg.exec, c.stream), "cudaGraphLaunch")) return PEVSL_ERR_CUDA;
  for (const IlGroup &G : fg.groups)
    if ((st = il_unpack_group(G, jobs.data()))) return st;
  for (int e = 0; e < ne && !st; e++)
    if (!fg.grouped[(size_t)e])
      st = memcpy_async(jobs[e].y, staged[e].y, sizeof(double) * (size_t)jobs[e].A->nrows);
  return st;
}

/* One CGS_DGKS (SRC/miscla.c:211-240) of v against V(:, 0:k).  On entry the
 * device slot S_NRM0 holds ||v||; on exit S_NRM holds the final norm.  The
 * second pass runs only if the first kept at most 1/sqrt(2) of the norm,
 * decided on the device. */
int cgs_dgks(const double *V, long ldv, int k, double *v, long n) {
  Ctx &c = ctx();
  double *w = (double *)ws(WS_SMALL, sizeof(double) * (size_t)(k + 1));
  if (!w) return PEVSL_ERR_NOMEM;
  int *run2 = c.dflag + F_PASS2;
  if (gemvT(n, k, V, ldv, v, w, nullptr)) return PEVSL_ERR_CUDA;
  if (gemv_sub_nrm(n, k, V, ldv, w, v, c.dscal + S_NRM, nullptr, run2, c.dscal + S_NRM0, kEta))
    return PEVSL_ERR_CUDA;
  if (gemvT(n, k, V, ldv, v, w, run2)) return PEVSL_ERR_CUDA;
  return gemv_sub_nrm(n, k, V, ldv, w, v, c.dscal + S_NRM, run2, nullptr, nullptr, kEta);
}

long round_ld(long n) { return (n + 31) / 32 * 32; }

}  // namespace

extern "C" {

/* Filter-kernel counters since the last reset: launches of the fused
 * Chebyshev degree kernel inside pEVSL_ChebLanNr, their algorithmic bytes,
 * and the device time of the filter applications that contain them (CUDA
 * events around each application, so launch gaps are included). */
void pEVSL_B200_FilterCounters(uint64_t *launches, double *bytes, double *ms) {
  if (launches) *launches = g_filter_launches;
  if (bytes) *bytes = g_filter_bytes;
  if (ms) *ms = g_filter_ms;
}

void pEVSL_B200_ResetFilterCounters(void) {
  g_filter_launches = 0;
  g_filter_persistent = 0;
  g_filter_bytes = 0.0;
  g_filter_ms = 0.0;
}

/* y = p(A) v (pEVSL_ChebAv, SRC/chebpol.c:509-574) on device or managed
 * vectors of length pevsl->n.  Extension entry point: the reference keeps
 * ChebAv internal. */
int pEVSL_B200_ChebAv(pevsl_Data *pevsl, pevsl_Polparams *pol, const double *v, double *y) {
  if (ensure()) return PEVSL_ERR_CUDA;
  matrix_window(pevsl_builtin_A(pevsl));
  const long n = pevsl->n;
  double *w3 = (double *)ws(WS_CHEB, sizeof(double) * 3 * (size_t)n);
  if (!w3) return PEVSL_ERR_NOMEM;
  int st = cheb_apply(pevsl, pol, v, y, w3, n);
  if (!st) st = sync();
  return st;
}

/* ================================================================ KPM DOS */

/* host doubles without exceptions, which must not leave a C entry */
struct HostBuf {
  double *p = nullptr;
  size_t n = 0;
  bool reserve(size_t want) {
    if (want <= n && p) return true;
    free(p);
    p = (double *)malloc(sizeof(double) * (want ? want : 1));
    n = p ? want : 0;
    return p != nullptr;
  }
  ~HostBuf() { free(p); }
};

static constexpr int kKpmChunk = 64;

int pEVSL_Kpmdos(pevsl_Data *pevsl, int Mdeg, int damping, int nvec, double *intv, int ngroups,
                 int groupid, MPI_Comm gl_comm, double *mu, double *ecnt) {
  const double t0 = pevsl_now();
  if (ensure()) return PEVSL_ERR_CUDA;
  if (pevsl_check_intv(intv, stdout) < 0) return -1;
  const long n = pevsl->n;
  const double aa = PEVSL_MAX(intv[0], intv[2]), bb = PEVSL_MIN(intv[1], intv[3]);
  if (intv[0] < intv[2] || intv[1] > intv[3]) {
    fprintf(stdout, " warning: interval (%e, %e) is adjusted to (%e, %e)\n", intv[0], intv[1],
            aa, bb);
  }
  const double ctr = (intv[3] + intv[2]) / 2.0, wid = (intv[3] - intv[2]) / 2.0;
  const double beta1 = acos(PEVSL_MAX(-1.0 + DBL_EPSILON, (aa - ctr) / wid));
  const double beta2 = acos(PEVSL_MIN(1.0 - DBL_EPSILON, (bb - ctr) / wid));
  double *jac = (double *)malloc(sizeof(double) * (size_t)(Mdeg + 1));
  if (!jac) return PEVSL_ERR_NOMEM;
  pevsl_dampcf(Mdeg, damping, jac);
  jac[0] = 1.0;
  memset(mu, 0, sizeof(double) * (size_t)(Mdeg + 1));
  double tcnt = 0.0;
  int vec_start = 0, vec_end = nvec;
  if (ngroups > 1) pEVSL_Part1d(nvec, ngroups, &groupid, &vec_start, &vec_end, 1);
  /* counter-based Gaussian stream: a group starts at its first vector's
   * draw, so the groups' vectors are exactly one process's nvec vectors and
   * the summed moments equal the one-group moments (the C library stream is
   * per process, as the reference's per-rank srand) */
  if (ngroups > 1 && pevsl_rng_mode() == PEVSL_RNG_GAUSS && vec_start > 0)
    pevsl_rng_take((uint64_t)vec_start);
  pevsl_devcsr *A = pevsl_builtin_A(pevsl);
  int st = 0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, ctx().stream);
  const bool gen = pevsl->ifGenEv != 0;
  const bool mixed = !gen && A && pevsl_inst_of(pevsl)->precision == PEVSL_PREC_MIXED;
  if (mixed) st = csr_make_fp32(A);
  if (gen) {
    /* generalized problem: one vector at a time with B-solves */
    if (!st)
      st = pevsl_gen_kpm_moments(pevsl, Mdeg, jac, ctr, wid, beta1, beta2, vec_start, vec_end, mu,
                                 &tcnt);
  } else if (A && mixed && !st) {
    /* FP32 moments: blocks of up to 64 vectors drawn and normalised in FP64,
     * then rounded to FP32; FP32 recurrence and dots, one launch per degree */
    const int smax = 64;
    for (int m0 = vec_start; m0 < vec_end && !st; m0 += smax) {
      const int s = vec_end - m0 < smax ? vec_end - m0 : smax;
      const int ld = s;
      const size_t blk = (size_t)n * (size_t)ld;
      double *X = (double *)ws(WS_KPM, sizeof(double) * 4 * blk);
      double *mom = (double *)ws(WS_MOM, sizeof(double) * (size_t)(Mdeg + 1) * (size_t)s);
      double *nrm2 = (double *)ws(WS_SMALL, sizeof(double) * 64);
      double *hmom = (double *)malloc(sizeof(double) * (size_t)(Mdeg + 1) * (size_t)s);
      if (!X || !mom || !nrm2 || !hmom) {
        free(hmom);
        st = PEVSL_ERR_NOMEM;
        break;
      }
      double *V0d = X;
      float *V0 = (float *)(X + blk), *B[3] = {V0 + blk, V0 + 2 * blk, V0 + 3 * blk};
      st = pevsl_rand_block_dev(V0d, (int)n, s, ld);
      if (!st) st = block_colnorm2(n, s, ld, V0d, nrm2);
      if (!st) st = block_normalize(n, s, ld, V0d, nrm2);
      if (!st) st = cvt_f64_f32((long)blk, V0d, V0);
      for (int k = 0; k < Mdeg && !st; k++) {
        const double sc = (k == 0 ? 1.0 : 2.0) / wid;
        const float *Xk = k == 0 ? V0 : B[(k - 1) % 3];
        const float *Xkm1 = k == 0 ? nullptr : (k == 1 ? V0 : B[(k - 2) % 3]);
        st = kpm_step32(A, s, ld, Xk, Xkm1, B[k % 3], V0, ctr, sc, mom + (size_t)k * s);
      }
      if (!st) st = memcpy_async(hmom, mom, sizeof(double) * (size_t)Mdeg * (size_t)s);
      if (!st) st = sync();
      pevsl->stats->n_mvA += (size_t)Mdeg * (size_t)s;
      for (int c = 0; c < s && !st; c++) {
        mu[0] += jac[0];
        tcnt -= jac[0] * (beta2 - beta1);
        for (int k = 0; k < Mdeg; k++) {
          const int k1 = k + 1;
          const double t = hmom[(size_t)k * s + c] * 2.0 * jac[k1];
          mu[k1] += t;
          tcnt -= t * (sin(k1 * beta2) - sin(k1 * beta1)) / k1;
        }
      }
      free(hmom);
    }
  } else if (A && !st) {
    /* groups of vectors, row-interleaved; one launch per degree.  With
     * c_k = <v_k, v_0>, T_{2k} = 2 T_k^2 - 1 and T_{2k+1} = 2 T_{k+1} T_k -
     * T_1 give c_{2k} = 2 <v_k, v_k> - c_0 and c_{2k+1} = 2 <v_{k+1}, v_k> -
     * c_1, so half the degrees do. */
    const int smax = kpm_group(A, vec_end - vec_start), steps = (Mdeg + 1) / 2;
    HostBuf hmom;
    for (int m0 = vec_start; m0 < vec_end && !st; m0 += smax) {
      const int s = PEVSL_MIN(smax, vec_end - m0), ld = (s + 1) / 2 * 2;
      const size_t nmom = 4 * (size_t)ld * (size_t)(steps + 1);
      const size_t blk = (size_t)n * (size_t)ld, np = (size_t)kpm_blocks(A, s) * 2 * (size_t)ld;
      double *X = (double *)ws(WS_KPM, sizeof(double) * 2 * blk);
      /* the blocks' sums of up to kKpmChunk steps, then added up: 39 MB for 64
       * vectors, however many moments */
      const int chunk = PEVSL_MIN(PEVSL_MAX(steps, 1), kKpmChunk);
      double *part = (double *)ws(WS_PART, sizeof(double) * np * (size_t)chunk);
      /* per step, and first for the start vectors */
      double *mom = (double *)ws(WS_MOM, sizeof(double) * nmom);
      double *nrm2 = (double *)ws(WS_SMALL, sizeof(double) * 64);
      if (!X || !part || !mom || !nrm2 || !hmom.reserve(nmom)) {
        st = PEVSL_ERR_NOMEM;
        break;
      }
      double *B[2] = {X, X + blk};
      if (s < ld)
        st = fail(cudaMemset2DAsync(X + s, sizeof(double) * (size_t)ld, 0, sizeof(double), (size_t)n,
                                    ctx().stream),
                  "cudaMemset2DAsync");
      if (!st) st = pevsl_rand_block_dev(X, (int)n, s, ld);
      if (!st) st = block_colnorm2(n, s, ld, X, nrm2);
      if (!st) st = block_normalize(n, s, ld, X, nrm2);
      if (!st) st = kpm_start(A, s, X, part);
      if (!st) st = kpm_reduce(A, s, 1, part, mom);
      for (int k = 0; k < steps && !st; k++) {
        const int at = k % chunk;
        st = kpm_step(A, s, B[k % 2], k > 0 ? B[(k + 1) % 2] : nullptr, B[(k + 1) % 2], ctr,
                      (k == 0 ? 1.0 : 2.0) / wid, part + np * (size_t)at);
        if (!st && (at == chunk - 1 || k == steps - 1))
          st = kpm_reduce(A, s, at + 1, part, mom + 4 * (size_t)ld * (size_t)(k - at + 1));
      }
      if (!st) st = memcpy_async(hmom.p, mom, sizeof(double) * nmom);
      if (!st) st = sync();
      pevsl->stats->n_mvA += (size_t)steps * (size_t)s;
      /* accumulate exactly as the reference: vector by vector, degree by degree */
      for (int c = 0; c < s && !st; c++) {
        mu[0] += jac[0];
        tcnt -= jac[0] * (beta2 - beta1);
        /* c_0 of the start vector as block_normalize left it, one up to
         * rounding, and known as well as the products it is subtracted from */
        const double *h1 = hmom.p + 4 * (size_t)ld; /* the first step's */
        const long double c0 = (long double)hmom.p[4 * (size_t)c] + hmom.p[4 * (size_t)c + 1];
        const long double c1 = steps > 0 ? (long double)h1[4 * (size_t)c + 2] + h1[4 * (size_t)c + 3] : 0;
        for (int k = 0; k < Mdeg; k++) {
          const int k1 = k + 1;
          const double *d = h1 + 4 * ((size_t)(k / 2) * ld + c);
          const double ck = (double)(k == 0       ? c1
                                     : k1 % 2 ? 2.0L * ((long double)d[2] + d[3]) - c1
                                              : 2.0L * ((long double)d[0] + d[1]) - c0);
          const double t = ck * 2.0 * jac[k1];
          mu[k1] += t;
          tcnt -= t * (sin(k1 * beta2) - sin(k1 * beta1)) / k1;
        }
      }
    }
  } else if (!st) {
    /* user matvec: one vector at a time, as the reference */
    double *buf = (double *)ws(WS_KPM, sizeof(double) * 4 * (size_t)n);
    double *hdot = (double *)malloc(sizeof(double) * (size_t)(Mdeg + 1));
    double *ddot_ = (double *)ws(WS_MOM, sizeof(double) * (size_t)(Mdeg + 1));
    if (!buf || !hdot || !ddot_) st = PEVSL_ERR_NOMEM;
    for (int m = vec_start; m < vec_end && !st; m++) {
      double *v = buf, *vkm1 = buf + n, *vk = buf + 2 * n, *vkp1 = buf + 3 * n, *tmp;
      st = pevsl_rand_vector_dev(v, (int)n);
      if (!st) st = vnrm2(n, v, ctx().dscal + S_TMP0);
      const double *h = st ? nullptr : fetch_scalars(S_TMP0, 1);
      if (!h) {
        st = st ? st : PEVSL_ERR_CUDA;
        break;
      }
      const double tn = h[0];
      if (!st) st = vscal(v, n, 1.0 / tn);
      if (!st) st = vcopy(v, vk, n);
      if (!st) st = vfill(vkm1, n, 0.0);
      for (int k = 0; k < Mdeg && !st; k++) {
        const double sc = (k == 0 ? 1.0 : 2.0) / wid;
        st = apply_A(pevsl, vk, vkp1);
        if (!st) st = vaxpy(n, -ctr, vk, vkp1);
        if (!st) st = vscal(vkp1, n, sc);
        if (!st) st = vaxpy(n, -1.0, vkm1, vkp1);
        tmp = vkm1;
        vkm1 = vk;
        vk = vkp1;
        vkp1 = tmp;
        if (!st) st = vdot(n, vk, v, ddot_ + k);
      }
      if (!st) st = memcpy_async(hdot, ddot_, sizeof(double) * (size_t)Mdeg);
      if (!st) st = sync();
      if (st) break;
      mu[0] += jac[0];
      tcnt -= jac[0] * (beta2 - beta1);
      for (int k = 0; k < Mdeg; k++) {
        const int k1 = k + 1;
        const double t = hdot[k] * 2.0 * jac[k1];
        mu[k1] += t;
        tcnt -= t * (sin(k1 * beta2) - sin(k1 * beta1)) / k1;
      }
    }
    free(hdot);
  }
  cudaEventRecord(e1, ctx().stream);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  pevsl_inst_of(pevsl)->phase_ms[1] = ms;
  free(jac);
  if (st) return st;
  if (ngroups > 1) {
    /* the groups' partial sums (SRC/kpmdos.c:160-176): through the
     * instance's reduction (one process per GPU) when one is installed,
     * else MPI on gl_comm */
    pevsl_inst *inst = pevsl_inst_of(pevsl);
    double *mu_g = (double *)malloc(sizeof(double) * (size_t)(Mdeg + 2));
    if (!mu_g) return PEVSL_ERR_NOMEM;
    if (inst->group_reduce) {
      memcpy(mu_g, mu, sizeof(double) * (size_t)(Mdeg + 1));
      mu_g[Mdeg + 1] = tcnt;
      inst->group_reduce(mu_g, Mdeg + 2, inst->group_reduce_ctx);
      memcpy(mu, mu_g, sizeof(double) * (size_t)(Mdeg + 1));
      tcnt = mu_g[Mdeg + 1];
    } else {
      double tcnt_g = 0.0;
      MPI_Allreduce(mu, mu_g, Mdeg + 1, MPI_DOUBLE, MPI_SUM, gl_comm);
      MPI_Allreduce(&tcnt, &tcnt_g, 1, MPI_DOUBLE, MPI_SUM, gl_comm);
      memcpy(mu, mu_g, sizeof(double) * (size_t)(Mdeg + 1));
      tcnt = tcnt_g;
    }
    free(mu_g);
  }
  const double t = 1.0 / (((double)nvec) * M_PI);
  for (int k = 0; k <= Mdeg; k++) mu[k] *= t;
  tcnt *= t * ((double)pevsl->N);
  *ecnt = tcnt;
  pevsl->stats->t_dos = pevsl_now() - t0;
  return 0;
}

/* ================================================================ Lanczos DOS */

/* Host threads for the per-slice host work of a lockstep group (the
 * tridiagonal eigenproblems of the convergence tests and the Ritz
 * extraction): PEVSL_B200_HOST_THREADS caps them (1: the calling thread
 * only; default: every hardware thread). */
static unsigned host_threads() {
  static unsigned v = 0;
  if (!v) {
    const char *e = getenv("PEVSL_B200_HOST_THREADS");
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const int r = e ? atoi(e) : 0;
    v = r >= 1 ? std::min((unsigned)r, hw) : hw;
  }
  return v;
}

/* f(0), ..., f(m-1) on up to host_threads() threads, this one included,
 * when worth is set; else in order on this thread.  f must be host-only
 * code (no CUDA call) that writes nothing another index reads. */
extern "C++" {
template <class F>
static void host_parallel(size_t m, bool worth, F f) {
  const size_t nt = std::min<size_t>(m, host_threads());
  if (!worth || nt <= 1) {
    for (size_t i = 0; i < m; i++) f(i);
    return;
  }
  std::atomic<size_t> next{0};
  auto work = [&]() {
    for (size_t i = next.fetch_add(1); i < m; i = next.fetch_add(1)) f(i);
  };
  std::vector<std::thread> th;
  for (size_t t = 1; t < nt; t++) {
    try {
      th.emplace_back(work);
    } catch (...) {
      break; /* no more threads: this one does the rest */
    }
  }
  work();
  for (auto &x : th) x.join();
}
}  // extern "C++"

/* Lanczos steps of S <= kMaxBatch independent runs in lockstep, queued
 * without a host synchronisation: alpha and beta stay on the device, where
 * the next step reads them, and the host reads all steps at once.  (A
 * breakdown therefore shows only then; what was queued past it is dropped.
 * A user operator, whose call waits for the GPU anyway, must not see such
 * steps' vectors, which were divided by nearly nothing: with one, a step is
 * queued only when the one before has been looked at.)  The callers count
 * the products of the built-in operator, those of the dropped steps apart.
 * Run s has its basis at V[s] (leading dimension ld).  Per run the kernels
 * and their decompositions are those of a single run, so each run's values
 * are the bits it has alone. */
struct LanRuns {
  pevsl_Data *pevsl;
  int S;
  long n, ld;
  int maxk;                /* columns of a basis */
  double *V[kMaxBatch];
  double *hist, *nrm0, *w; /* [step][alpha, beta][S]; norms; CGS coefficients */
  double *alpha(int step) const { return hist + 2 * (size_t)step * S; }
  double *beta(int step) const { return alpha(step) + S; }
};

static int lan_init(LanRuns &R, pevsl_Data *pevsl, int S, double *V, long stride, long n, long ld,
                    int maxk) {
  R.pevsl = pevsl;
  R.S = S;
  R.n = n;
  R.ld = ld;
  R.maxk = maxk;
  for (int s = 0; s < S; s++) R.V[s] = V + (size_t)s * (size_t)stride;
  const size_t h = 2 * (size_t)maxk * S;
  R.hist = (double *)ws(WS_LAN, sizeof(double) * (h + S + (size_t)S * (size_t)(maxk + 1)));
  if (!R.hist) return PEVSL_ERR_NOMEM;
  R.nrm0 = R.hist + h;
  R.w = R.nrm0 + S;
  return 0;
}

/* step k: V(:, k+1) from V(:, k) and V(:, k-1); prev: subtract beta(k-1)
 * V(:, k-1) */
static int lan_step(LanRuns &R, int k, bool prev) {
  const int S = R.S;
  const unsigned all = (1u << S) - 1u;
  const BLen len = blen_uniform(R.n, R.ld, S);
  CPtrs v{}, vm{}, vc{}, base{};
  VPtrs vn{};
  for (int s = 0; s < S; s++) {
    base.p[s] = R.V[s];
    v.p[s] = R.V[s] + (size_t)k * R.ld;
    vm.p[s] = prev ? v.p[s] - R.ld : nullptr;
    vn.p[s] = R.V[s] + (size_t)(k + 1) * R.ld;
    vc.p[s] = vn.p[s];
  }
  int *flag = ctx().gflag;
  int st = 0;
  if (pevsl_devcsr *A = pevsl_builtin_A(R.pevsl)) {
    st = spmv_batch(A, S, v, vn);
  } else {
    for (int s = 0; s < S && !st; s++) st = apply_A(R.pevsl, v.p[s], vn.p[s]);
  }
  if (!st)
    st = prev ? b_axpy_dev_dot(len, S, R.beta(k - 1), -1.0, vm, vn, v, R.alpha(k))
              : b_dot(len, S, v, vc, R.alpha(k), FIN_ID, all);
  if (!st) st = b_axpy_dev_nrm2(len, S, R.alpha(k), v, vn, R.nrm0, all);
  const long ldw = R.maxk + 1;
  if (!st) st = b_gemvT(len, S, k + 1, base, vc, R.w, ldw, nullptr, all);
  if (!st)
    st = b_gemv_sub_nrm(len, S, k + 1, base, R.w, ldw, vn, R.beta(k), nullptr, flag, R.nrm0, kEta, all);
  if (!st) st = b_gemvT(len, S, k + 1, base, vc, R.w, ldw, flag, all);
  if (!st)
    st = b_gemv_sub_nrm(len, S, k + 1, base, R.w, ldw, vn, R.beta(k), flag, nullptr, nullptr, kEta, all);
  if (!st) st = b_scal_inv_dev(len, S, R.beta(k), vn);
  return st;
}

/* one Lanczos run of pEVSL_LanDosG (SRC/landos.c:134-262): v_0 = vinit
 * normalised, maxit steps with full reorthogonalisation; the tridiagonal
 * matrix into dT, eT */
extern "C++" {
template <class Draw>
static int landos_lanczos(pevsl_Data *pevsl, int maxit, double *V, long ld, const double *vinit,
                          long n, double *dT, double *eT, Draw draw) {
  Ctx &c = ctx();
  int st = vnrm2(n, vinit, c.dscal + S_TMP0);
  const double *h = st ? nullptr : fetch_scalars(S_TMP0, 1);
  if (!h) return st ? st : PEVSL_ERR_CUDA;
  const double tinv = 1.0 / h[0];
  if (!st) st = vcopy(vinit, V, n);
  if (!st) st = vscal(V, n, tinv);
  double wn = 0.0, beta = 0.0;
  int nwn = 0;
  for (int k = 0; k < maxit && !st; k++) {
    double *v = V + (size_t)k * ld, *vnew = V + (size_t)(k + 1) * ld;
    st = apply_A(pevsl, v, vnew);
    if (!st && k > 0) st = vaxpy(n, -beta, V + (size_t)(k - 1) * ld, vnew);
    if (!st) st = vdot(n, v, vnew, c.dscal + S_ALPHA);
    if (!st) st = vaxpy_dev_nrm2(n, c.dscal + S_ALPHA, v, vnew, c.dscal + S_NRM0);
    if (!st) st = cgs_dgks(V, ld, k + 1, vnew, n);
    if (!st) st = memcpy_async(c.hscal + S_ALPHA, c.dscal + S_ALPHA, sizeof(double) * 4);
    if (!st) st = sync();
    if (st) break;
    const double alpha = c.hscal[S_ALPHA];
    beta = c.hscal[S_NRM];
    dT[k] = alpha;
    wn += fabs(alpha) + 2.0 * beta;
    nwn += 3;
    if (beta * nwn < orthTol * wn) {
      st = draw(vnew);
      if (!st) st = vnrm2(n, vnew, c.dscal + S_NRM0);
      if (!st) st = cgs_dgks(V, ld, k + 1, vnew, n);
      const double *hb = st ? nullptr : fetch_scalars(S_NRM, 1);
      if (!hb) return st ? st : PEVSL_ERR_CUDA;
      st = vscal(vnew, n, 1.0 / hb[0]);
      beta = 0.0;
    } else {
      st = vscal(vnew, n, 1.0 / beta);
    }
    eT[k] = beta;
  }
  return st;
}

}  // extern "C++"

/* the S runs of a group in lockstep from the start vectors vinit(:, 0:S)
 * (unchanged); *good: how many of them, from the first on, did not break down.
 * (The next one draws another start vector, so it and those after it are to
 * be run one by one.) */
static int landos_lockstep(pevsl_Data *pevsl, int S, int maxit, double *V, long ld,
                           const double *vinit, long n, double *dT, double *eT, int *good) {
  *good = S;
  LanRuns R;
  int st = lan_init(R, pevsl, S, V, ld * (maxit + 1), n, ld, maxit + 1);
  CPtrs x{};
  VPtrs v0{};
  for (int s = 0; s < S && !st; s++) {
    st = vcopy(vinit + (size_t)s * ld, R.V[s], n);
    x.p[s] = R.V[s];
    v0.p[s] = R.V[s];
  }
  const BLen len = blen_uniform(n, ld, S);
  if (!st) st = b_dot(len, S, x, x, R.nrm0, FIN_SQRT, (1u << S) - 1u);
  if (!st) st = b_scal_inv_dev(len, S, R.nrm0, v0);
  for (int k = 0; k < maxit && !st; k++) st = lan_step(R, k, k > 0);
  HostBuf hist;
  if (!st && !hist.reserve(2 * (size_t)maxit * S)) st = PEVSL_ERR_NOMEM;
  const double *h = hist.p;
  if (!st) st = memcpy_async(hist.p, R.hist, sizeof(double) * 2 * (size_t)maxit * S);
  if (!st) st = sync();
  for (int s = 0; s < *good && !st; s++) {
    double wn = 0.0;
    int nwn = 0;
    for (int k = 0; k < maxit; k++) {
      const double alpha = h[2 * (size_t)k * S + s], beta = h[(2 * (size_t)k + 1) * S + s];
      dT[(size_t)s * maxit + k] = alpha;
      eT[(size_t)s * maxit + k] = beta;
      wn += fabs(alpha) + 2.0 * beta;
      nwn += 3;
      if (beta * nwn < orthTol * wn) *good = s;
    }
  }
  if (!st) pevsl->stats->n_mvA += (size_t)maxit * (size_t)*good;
  return st;
}

static constexpr size_t kKeepBasis = (size_t)1 << 30;

int pEVSL_LanDosG(pevsl_Data *pevsl, const int nvec, int msteps, int npts, double *xdos,
                  double *ydos, double *neig, double *intv, int ngroups, int groupid,
                  MPI_Comm gl_comm) {
  if (ensure()) return PEVSL_ERR_CUDA;
  const double t0 = pevsl_now();
  const long n = pevsl->n, ld = round_ld(n);
  const int maxit = msteps < pevsl->N ? msteps : pevsl->N;
  int vec_start = 0, vec_end = nvec;
  if (ngroups > 1) pEVSL_Part1d(nvec, ngroups, &groupid, &vec_start, &vec_end, 1);
  /* runs in lockstep: up to kMaxBatch, their bases within 4 GB and their
   * eigenvectors of T within 256 MB of host memory, the groups about equal;
   * fewer where there is no memory for as many; one at a time with B-solves
   * or a user operator, and where every run breaks down at its N-th step */
  const double basis = 8.0 * (double)ld * (maxit + 1), evec = 8.0 * maxit * (double)maxit;
  const int nrun = PEVSL_MAX(vec_end - vec_start, 0);
  const bool ahead = !pevsl->ifGenEv && pevsl_builtin_A(pevsl) && maxit < pevsl->N;
  int lock = !ahead ? 1 : (int)PEVSL_MIN((double)kMaxBatch, PEVSL_MAX(1.0, PEVSL_MIN(4e9 / basis, 256e6 / evec)));
  const size_t held = ctx().wsz[WS_BASIS];
  double *V = nullptr, *vinit = nullptr;
  for (;; lock /= 2) {
    const int ngr = PEVSL_MAX(1, (nrun + lock - 1) / lock);
    lock = PEVSL_MAX(1, (nrun + ngr - 1) / ngr);
    const size_t vb = sizeof(double) * (size_t)ld * (size_t)(maxit + 1) * (size_t)lock;
    const size_t ib = sizeof(double) * (size_t)ld * (size_t)(lock + 1);
    V = (double *)(lock > 1 ? ws_try(WS_BASIS, vb) : ws(WS_BASIS, vb));
    vinit = !V ? nullptr : (double *)(lock > 1 ? ws_try(WS_LANV, ib) : ws(WS_LANV, ib));
    if (vinit || lock == 1) break;
  }
  double *y = (double *)calloc((size_t)npts, sizeof(double));
  int *ind = (int *)malloc(sizeof(int) * (size_t)npts);
  double *dT = (double *)malloc(sizeof(double) * (size_t)maxit * (size_t)lock);
  double *eT = (double *)malloc(sizeof(double) * (size_t)maxit * (size_t)lock);
  double *EvalT = (double *)malloc(sizeof(double) * (size_t)maxit * (size_t)lock);
  double *EvecT = (double *)malloc(sizeof(double) * (size_t)maxit * (size_t)maxit * (size_t)lock);
  int st = (!V || !vinit || !y || !ind || !dT || !eT || !EvalT || !EvecT) ? PEVSL_ERR_NOMEM : 0;
  const double lm = intv[2], lM = intv[3];
  const double aa = PEVSL_MAX(intv[0], intv[2]), bb = PEVSL_MIN(intv[1], intv[3]);
  const int M = PEVSL_MIN(msteps, 30);
  const double H = (lM - lm) / (M - 1);
  const double sigma = H / sqrt(8 * log(1.25)) * pevsl->sigma_mult;
  const double sigma2 = 2 * sigma * sigma;
  const double width = sigma * sqrt(-2.0 * log(1e-08));
  if (!st) linspace(aa, bb, npts, xdos);
  for (int m0 = vec_start; m0 < vec_end && !st; m0 += lock) {
    const int S = PEVSL_MIN(lock, vec_end - m0);
    /* the group's start vectors in draw order; a breakdown restart takes the
     * next one, as in runs one after the other */
    int drawn = 0, next = 0, good = 0;
    for (; drawn < S && !st; drawn++) st = pevsl_rand_vector_dev(vinit + (size_t)drawn * ld, (int)n);
    auto draw = [&](double *v) -> int {
      return next < drawn ? vcopy(vinit + (size_t)next++ * ld, v, n) : pevsl_rand_vector_dev(v, (int)n);
    };
    if (!st && ahead) st = landos_lockstep(pevsl, S, maxit, V, ld, vinit, n, dT, eT, &good);
    next = good;
    double *one = vinit + (size_t)lock * ld;
    for (int s = good; s < S && !st; s++) {
      st = draw(one);
      if (!st)
        st = pevsl->ifGenEv
                 ? pevsl_gen_landos_lanczos(pevsl, maxit, one, dT + (size_t)s * maxit, eT + (size_t)s * maxit)
                 : landos_lanczos(pevsl, maxit, V, ld, one, n, dT + (size_t)s * maxit,
                                  eT + (size_t)s * maxit, draw);
    }
    if (st) break;
    int es[kMaxBatch] = {0};
    host_parallel((size_t)S, maxit >= 30, [&](size_t s) {
      es[s] = pevsl_tridiag_eig(maxit, dT + s * maxit, eT + s * maxit, EvalT + s * maxit,
                                EvecT + s * (size_t)maxit * maxit);
    });
    for (int s = 0; s < S && !st; s++) {
      if (es[(size_t)s]) {
        st = PEVSL_ERR_EIG;
        break;
      }
      const double *ev = EvecT + (size_t)s * maxit * maxit;
      for (int i = 0; i < maxit; i++) {
        const double g2 = ev[(size_t)i * maxit] * ev[(size_t)i * maxit];
        const double th = EvalT[(size_t)s * maxit + i];
        int np = 0;
        for (int j = 0; j < npts; j++)
          if (fabs(xdos[j] - th) < width) ind[np++] = j;
        for (int j = 0; j < np; j++)
          y[ind[j]] += g2 * exp(-((xdos[ind[j]] - th) * (xdos[ind[j]] - th)) / sigma2);
      }
    }
  }
  if (!st && ngroups > 1) {
    double *yg = (double *)malloc(sizeof(double) * (size_t)npts);
    MPI_Allreduce(y, yg, npts, MPI_DOUBLE, MPI_SUM, gl_comm);
    memcpy(y, yg, sizeof(double) * (size_t)npts);
    free(yg);
  }
  if (!st) {
    const double scaling = 1.0 / (nvec * sqrt(sigma2 * M_PI));
    for (int j = 0; j < npts; j++) y[j] *= scaling;
    memcpy(ydos, y, sizeof(double) * (size_t)npts);
    pevsl_simpson(xdos, y, npts);
    *neig = y[npts - 1] * pevsl->N;
  }
  free(y);
  free(ind);
  free(dT);
  free(eT);
  free(EvalT);
  free(EvecT);
  /* bases of several runs beyond 1 GB go back, unless the workspace was as
   * large before */
  if (lock > 1 && held < kKeepBasis && ctx().wsz[WS_BASIS] > kKeepBasis) ws_free(WS_BASIS);
  pevsl->stats->t_dos = pevsl_now() - t0;
  return st;
}

/* ================================================================ bounds */

int pEVSL_LanTrbounds(pevsl_Data *pevsl, int lanm, int maxit, double tol, pevsl_Parvec *vinit,
                      int bndtype, double *lammin, double *lammax, FILE *fstats) {
  if (ensure()) return PEVSL_ERR_CUDA;
  const double t0 = pevsl_now();
  if (pevsl->ifGenEv) {
    const int st = pevsl_gen_lantrbounds(pevsl, lanm, maxit, tol, vinit, bndtype, lammin, lammax,
                                         fstats);
    pevsl->stats->t_eigbounds += pevsl_now() - t0;
    pevsl_inst_of(pevsl)->phase_ms[0] = 1e3 * (pevsl_now() - t0);
    return st;
  }
  const int N = pevsl->N;
  const long n = pevsl->n, ld = round_ld(n);
  lanm = PEVSL_MIN(lanm, N);
  const int lanm1 = lanm + 1;
  if (lanm == N) maxit = PEVSL_MIN(maxit, N);
  const size_t L = (size_t)lanm1;
  double *V = (double *)ws(WS_BASIS, sizeof(double) * (size_t)ld * L);
  double *R2 = (double *)ws(WS_RITZ, sizeof(double) * (size_t)ld * 2);
  double *dY = (double *)ws(WS_RITZ2, sizeof(double) * L * 2 + sizeof(double) * L);
  double *T = (double *)calloc(L * L, sizeof(double));
  double *EvecT = (double *)calloc(L * L, sizeof(double));
  double *Rval = (double *)calloc(L, sizeof(double));
  double *hY = (double *)malloc(sizeof(double) * L * 2);
  if (!V || !R2 || !dY || !T || !EvecT || !Rval || !hY) {
    free(T);
    free(EvecT);
    free(Rval);
    free(hY);
    return PEVSL_ERR_NOMEM;
  }
  double *dS = dY + 2 * L; /* coefficients s of the restart step */
  Ctx &c = ctx();
  int st = 0, it = 0, trlen = 0;
  LanRuns R;
  st = lan_init(R, pevsl, 1, V, 0, n, ld, lanm1);
  HostBuf hist;
  if (!st && !hist.reserve(2 * L)) st = PEVSL_ERR_NOMEM;
  double lmin = 0.0, lmax = 0.0, s[3] = {0, 0, 0};
  if (fstats) fprintf(fstats, " LanTR for bounds: dim %d, maxits %d\n", lanm, maxit);
  if (!st) st = vcopy(vinit->data, V, n);
  if (!st) st = vnrm2(n, V, c.dscal + S_TMP0);
  const double *h0 = st ? nullptr : fetch_scalars(S_TMP0, 1);
  if (!h0) st = st ? st : PEVSL_ERR_CUDA;
  if (!st) st = vscal(V, n, 1.0 / h0[0]);
#define VC(j) (V + (size_t)(j) * ld)
  while (it < maxit && !st) {
    double wn = 0.0, beta = 0.0;
    int nwn = 0;
    int k = trlen > 0 ? trlen + 1 : 0;
    if (k + 5 > lanm1) {
      fprintf(stderr, "Krylov dim too small for this problem. Try a larger dim\n");
      st = PEVSL_ERR_ARG;
      break;
    }
    if (trlen > 0) {
      /* thick-restart step: arrowhead column of T (SRC/lantrbnd.c:150-223) */
      const int k1 = k - 1;
      double *v = VC(k1), *vnew = VC(k1 + 1);
      st = apply_A(pevsl, v, vnew);
      for (int i = 0; i < trlen; i++) {
        T[i * L + i] = Rval[i];
        wn += fabs(Rval[i]);
      }
      if (!st) st = vdot(n, v, vnew, c.dscal + S_TMP0);
      const double *hs = st ? nullptr : fetch_scalars(S_TMP0, 1);
      if (!hs) {
        st = st ? st : PEVSL_ERR_CUDA;
        break;
      }
      s[k1] = hs[0];
      if (!st) st = memcpy_async(dS, s, sizeof(double) * (size_t)k);
      if (!st) st = gemv_sub_nrm(n, k, V, ld, dS, vnew, c.dscal + S_NRM, nullptr, nullptr, nullptr,
                                 kEta);
      for (int i = 0; i < k1; i++) {
        T[trlen * L + i] = s[i];
        T[i * L + trlen] = s[i];
        wn += 2.0 * fabs(s[i]);
      }
      T[trlen * L + trlen] = s[k1];
      wn += fabs(s[k1]);
      const double *hb = st ? nullptr : fetch_scalars(S_NRM, 1);
      if (!hb) {
        st = st ? st : PEVSL_ERR_CUDA;
        break;
      }
      beta = hb[0];
      wn += 2.0 * beta;
      nwn += 3 * k;
      if (beta * nwn < orthTol * wn) {
        st = pevsl_rand_vector_dev(vnew, (int)n);
        if (!st) st = vnrm2(n, vnew, c.dscal + S_NRM0);
        if (!st) st = cgs_dgks(V, ld, k, vnew, n);
        const double *hb2 = st ? nullptr : fetch_scalars(S_NRM, 1);
        if (!hb2) {
          st = st ? st : PEVSL_ERR_CUDA;
          break;
        }
        st = vscal(vnew, n, 1.0 / hb2[0]);
        beta = 0.0;
      } else {
        st = vscal(vnew, n, 1.0 / beta);
      }
      T[k1 * L + k] = beta;
      T[k * L + k1] = beta;
    }
    /* the steps of this cycle, queued at once; then their alpha and beta are
     * read, and after a breakdown the steps past it are queued again */
    bool prev = k > 0;
    const bool ahead = pevsl_builtin_A(pevsl) != nullptr;
    const int kend = PEVSL_MIN(lanm, k + maxit - it);
    while (k < kend && !st) {
      const int k0 = k, m = ahead ? kend - k0 : 1;
      if (prev) st = memcpy_async(R.beta(k0 - 1), &beta, sizeof(double));
      for (int j = k0; j < k0 + m && !st; j++) st = lan_step(R, j, j > k0 || prev);
      if (!st) st = memcpy_async(hist.p, R.alpha(k0), sizeof(double) * 2 * (size_t)m);
      if (!st) st = sync();
      bool broke = false;
      for (int j = 0; j < m && !st && !broke; j++) {
        const double alpha = hist.p[2 * (size_t)j];
        beta = hist.p[2 * (size_t)j + 1];
        k++;
        it++;
        if (ahead) pevsl->stats->n_mvA++;
        T[(k - 1) * L + (k - 1)] = alpha;
        wn += fabs(alpha) + 2.0 * beta;
        nwn += 3;
        if (beta * nwn < orthTol * wn) {
          if (fstats) fprintf(fstats, "it %4d: Lucky breakdown, beta = %.15e\n", it, beta);
          double *vnew = VC(k);
          st = pevsl_rand_vector_dev(vnew, (int)n);
          if (!st) st = vnrm2(n, vnew, c.dscal + S_NRM0);
          if (!st) st = cgs_dgks(V, ld, k, vnew, n);
          const double *hb = st ? nullptr : fetch_scalars(S_NRM, 1);
          if (!hb) {
            st = st ? st : PEVSL_ERR_CUDA;
            break;
          }
          st = vscal(vnew, n, 1.0 / hb[0]);
          beta = 0.0;
          broke = true;
        }
        T[k * L + (k - 1)] = beta;
        T[(k - 1) * L + k] = beta;
      }
      prev = true;
    }
    if (st) break;
    double end[6];
    if (ritz_ends_ok(k)) {
      if ((st = ritz_ends(k, T, lanm1, dY, end))) break;
    } else {
      if (pevsl_dense_symeig(k, T, lanm1, EvecT, lanm1, Rval)) {
        st = PEVSL_ERR_EIG;
        break;
      }
      end[0] = Rval[0];
      end[1] = Rval[1];
      end[2] = k > 1 ? Rval[k - 2] : 0.0;
      end[3] = Rval[k - 1];
      end[4] = EvecT[k - 1];
      end[5] = EvecT[(size_t)(k - 1) * L + (k - 1)];
      memcpy(hY, EvecT, sizeof(double) * (size_t)k);
      memcpy(hY + k, EvecT + (size_t)(k - 1) * L, sizeof(double) * (size_t)k);
      if ((st = memcpy_async(dY, hY, sizeof(double) * 2 * (size_t)k))) break;
    }
    s[0] = beta * end[4];
    s[1] = beta * end[5];
    double t1, t2;
    if (bndtype <= 1) {
      t1 = fabs(s[0]);
      t2 = fabs(s[1]);
    } else {
      t1 = 2.0 * s[0] * s[0] / (end[1] - end[0]);
      t2 = 2.0 * s[1] * s[1] / (end[3] - end[2]);
    }
    lmin = end[0] - t1;
    lmax = end[3] + t2;
    /* the two extreme Ritz vectors become V(:,0:2) */
    st = gemm_nn(n, k, 2, V, ld, dY, k, R2, ld);
    if (!st) st = vcopy(R2, VC(0), n);
    if (!st) st = vcopy(R2 + ld, VC(1), n);
    trlen = 2;
    Rval[0] = end[0];
    Rval[1] = end[3];
    if (fstats)
      fprintf(fstats, "it %4d, k %3d: ritz %.15e %.15e, t1,t2 %e %e, res %.15e %.15e\n", it, k,
              Rval[0], Rval[1], t1, t2, fabs(s[0]), fabs(s[1]));
    if (t1 + t2 < tol * (fabs(lmin) + fabs(lmax))) break;
    memset(T, 0, sizeof(double) * L * L);
    if (!st) st = vcopy(VC(k), VC(trlen), n);
  }
#undef VC
  if (!st) st = sync();
  *lammin = lmin;
  *lammax = lmax;
  free(T);
  free(EvecT);
  free(Rval);
  free(hY);
  pevsl->stats->t_eigbounds += pevsl_now() - t0;
  pevsl_inst_of(pevsl)->phase_ms[0] = 1e3 * (pevsl_now() - t0);
  return st;
}

/* ================================================================ filtered Lanczos
 * pEVSL_ChebLanNr (SRC/cheblanNr.c:54-448) for a batch of slices that
 * advance in lockstep: at every Lanczos step one fused filter kernel per
 * degree serves all slices (the matrix is read once per degree), the
 * Gram-Schmidt kernels run batched, and one host read fetches every slice's
 * alpha and beta.  Each slice keeps its own basis, tridiagonal matrix,
 * convergence test and stop; a single slice is a batch of one and follows
 * exactly the reference's sequence of operations. */

struct SliceState {
  /* inputs: the slice and the problem it belongs to */
  double intv[4];
  const pevsl_Polparams *pol;
  int maxit;
  pevsl_Data *pevsl;
  pevsl_devcsr *A; /* built-in device CSR, or NULL for a user matvec */
  pevsl_Parvec *vinit;
  long n, ld;
  /* state */
  double *V;      /* basis, ld x (maxit+1) */
  double *dT, *eT, *EvalT;
  double wn, tr0, beta;
  int nwn, kdim, count, nconv;
  int active, done;
  /* outputs */
  int status, nev, its;
  int short_pairs; /* mixed form: refined pairs in [a, b] above tol */
  double *Lam, *res;
  pevsl_Parvecs *Rvec;
};

/* The host part of a slice's Ritz extraction: the eigenvalues of T again
 * and the eigenvectors of those >= bar.  Host arithmetic only, so the
 * slices of a group run it on host threads (host_parallel). */
struct RitzHost {
  int early = 0;  /* error that ends the extraction before any output */
  int sel_st = 0; /* the eigenvector step failed */
  int nsel = 0;
  int *sel = nullptr;
  double *Y = nullptr;
  double secs = 0.0;
};

static void ritz_host(SliceState *S, RitzHost *R) {
  const int kdim = S->kdim, count = S->count;
  const double bar = S->pol->bar;
  const double te = pevsl_now();
  /* eigenvalues again: the last convergence test may predate the last step
   * (a maxit exit), so more Ritz values than nconv may pass the bar test;
   * the outputs hold max(nconv, nsel) pairs */
  if (kdim > 0 && pevsl_tridiag_eig(kdim, S->dT, S->eT, S->EvalT, nullptr)) {
    R->early = PEVSL_ERR_EIG;
    return;
  }
  R->sel = (int *)malloc(sizeof(int) * (size_t)(kdim > 0 ? kdim : 1));
  if (!R->sel) {
    R->early = PEVSL_ERR_NOMEM;
    return;
  }
  for (int i = 0; i < count && kdim > 0; i++)
    if (S->EvalT[i] >= bar) R->sel[R->nsel++] = i;
  if (kdim > 0 && R->nsel > 0) {
    R->Y = (double *)malloc(sizeof(double) * (size_t)kdim * (size_t)R->nsel);
    if (!R->Y || pevsl_tridiag_eig_sel(kdim, S->dT, S->eT, S->EvalT, R->nsel, R->sel, R->Y))
      R->sel_st = PEVSL_ERR_EIG;
  }
  R->secs = pevsl_now() - te;
}

/* Ritz pairs of one finished slice (SRC/cheblanNr.c:339-413): eigenvectors
 * of T only for Ritz values >= bar (ritz_host, run before), U = V Y,
 * normalise, W = A U, Rayleigh quotients, interval check, residuals,
 * acceptance below tol.  Takes over R's buffers. */
static int ritz_extract(pevsl_Data *pevsl, SliceState *S, RitzHost *R, pevsl_Parvec *vinit,
                        long n, long ld, double tol) {
  Ctx &c = ctx();
  const int kdim = S->kdim;
  const double aa = S->intv[0], bb = S->intv[1];
  S->nev = 0;
  if (R->early) {
    free(R->sel);
    free(R->Y);
    R->sel = nullptr;
    R->Y = nullptr;
    return R->early;
  }
  int st = 0;
  const int nsel = R->nsel;
  int *sel = R->sel;
  double *Y = R->Y;
  R->sel = nullptr;
  R->Y = nullptr;
  const double te = pevsl_now();
  const int nout = PEVSL_MAX(S->nconv, nsel);
  S->Lam = (double *)malloc(sizeof(double) * (size_t)(nout > 0 ? nout : 1));
  S->res = (double *)malloc(sizeof(double) * (size_t)(nout > 0 ? nout : 1));
  S->Rvec = (pevsl_Parvecs *)calloc(1, sizeof(pevsl_Parvecs));
  if (!S->Lam || !S->res || !S->Rvec) {
    free(sel);
    free(Y);
    return PEVSL_ERR_NOMEM;
  }
  pEVSL_ParvecsDuplParvec(vinit, nout, (int)n, S->Rvec);
  if (nout > 0 && !S->Rvec->data) {
    free(sel);
    free(Y);
    return PEVSL_ERR_NOMEM;
  }
  if (kdim <= 0) {
    free(sel);
    free(Y);
    return 0;
  }
  st = R->sel_st;
  pevsl->stats->t_eig += R->secs + (pevsl_now() - te);
  if (!st && nsel > 0) {
    double *U = (double *)ws(WS_RITZ, sizeof(double) * (size_t)ld * (size_t)nsel);
    double *W = (double *)ws(WS_RITZ2, sizeof(double) * (size_t)ld * (size_t)nsel);
    double *dY = (double *)ws(WS_PART, sizeof(double) * (size_t)kdim * (size_t)nsel);
    double *dv = (double *)ws(WS_MOM, sizeof(double) * 3 * (size_t)nsel);
    double *hv = (double *)malloc(sizeof(double) * 3 * (size_t)nsel);
    if (!U || !W || !dY || !dv || !hv) st = PEVSL_ERR_NOMEM;
    if (!st) st = memcpy_async(dY, Y, sizeof(double) * (size_t)kdim * (size_t)nsel);
    if (!st) st = gemm_nn(n, kdim, nsel, S->V, ld, dY, kdim, U, ld);
    if (!st) st = vdot_cols(n, nsel, U, ld, U, ld, dv);
    if (!st) st = memcpy_async(hv, dv, sizeof(double) * (size_t)nsel);
    if (!st) st = sync();
    for (int j = 0; j < nsel && !st; j++) {
      const double t = sqrt(hv[j]);
      if (t == 0.0) {
        st = 2; /* zero eigenvector (SRC/cheblanNr.c:377-379) */
        break;
      }
      hv[nsel + j] = 1.0 / t;
    }
    if (!st) st = memcpy_async(dv + nsel, hv + nsel, sizeof(double) * (size_t)nsel);
    if (!st) st = vscal_cols(n, nsel, U, ld, dv + nsel);
    for (int j = 0; j < nsel && !st; j++) st = apply_A(pevsl, U + (size_t)j * ld, W + (size_t)j * ld);
    if (!st) st = vdot_cols(n, nsel, W, ld, U, ld, dv);
    if (!st) st = vaxpy_cols(n, nsel, dv, U, ld, W, ld);
    if (!st) st = vdot_cols(n, nsel, W, ld, W, ld, dv + 2 * nsel);
    if (!st) st = memcpy_async(hv, dv, sizeof(double) * 3 * (size_t)nsel);
    if (!st) st = sync();
    for (int j = 0; j < nsel && !st; j++) {
      const double lam = hv[j];
      if (lam < aa - DBL_EPSILON || lam > bb + DBL_EPSILON) continue;
      const double r0 = sqrt(hv[2 * nsel + j]);
      if (r0 < tol) {
        S->Lam[S->nev] = lam;
        S->res[S->nev] = r0;
        st = vcopy(U + (size_t)j * ld, S->Rvec->data + (size_t)S->nev * S->Rvec->ld, n);
        S->nev++;
      }
    }
    free(hv);
  }
  free(Y);
  free(sel);
  if (!st) st = sync();
  return st;
}

/* Ritz pairs of a slice whose Krylov basis came from the FP32 filter: one
 * FP64 filtered Rayleigh-Ritz sweep.  The FP32 recurrence leaves noise of
 * about 1e-6 relative in every direction of the basis, which Rayleigh-Ritz
 * on the basis alone cannot remove; one FP64 application of p(A) damps each
 * direction by p(lam_out)/p(lam_in), which is small except just outside the
 * slice, so those near-edge directions are taken into the subspace instead:
 * U = V Y for the Ritz values of p(A) >= guard * bar (guard < 1; the
 * reference keeps those >= bar, SRC/cheblanNr.c:350-365), P = p(A) U in
 * FP64 with unit columns, G = P'P, H = P'AP (gemm_tn), the pencil (H, G)
 * on the host (Cholesky dropping dependent columns), X = P Z, and the
 * reference's acceptance on the refined pairs (SRC/cheblanNr.c:366-405):
 * lam in [a, b] and ||A x - lam x|| < tol. */
static int ritz_refine(pevsl_Data *pevsl, SliceState *S, pevsl_Parvec *vinit, long n, long ld,
                       double tol, double guard, int passes) {
  pevsl_devcsr *A = pevsl_builtin_A(pevsl);
  const int kdim = S->kdim, count = S->count;
  const double bar = S->pol->bar, aa = S->intv[0], bb = S->intv[1];
  S->nev = 0;
  int m = 0, st = 0;
  int *sel = (int *)malloc(sizeof(int) * (size_t)(kdim > 0 ? kdim : 1));
  if (!sel) return PEVSL_ERR_NOMEM;
  if (kdim > 0 && pevsl_tridiag_eig(kdim, S->dT, S->eT, S->EvalT, nullptr)) st = PEVSL_ERR_EIG;
  int nbar = 0; /* Ritz values of p(A) above bar: the FP64 path's candidates */
  for (int i = 0; i < count && kdim > 0 && !st; i++) {
    if (S->EvalT[i] >= guard * bar) sel[m++] = i;
    if (S->EvalT[i] >= bar) nbar++;
  }
  S->short_pairs = nbar;
  S->Lam = (double *)malloc(sizeof(double) * (size_t)(m > 0 ? m : 1));
  S->res = (double *)malloc(sizeof(double) * (size_t)(m > 0 ? m : 1));
  S->Rvec = (pevsl_Parvecs *)calloc(1, sizeof(pevsl_Parvecs));
  if (!S->Lam || !S->res || !S->Rvec) st = PEVSL_ERR_NOMEM;
  if (st || m == 0) {
    if (S->Rvec) pEVSL_ParvecsDuplParvec(vinit, 0, (int)n, S->Rvec);
    free(sel);
    return st;
  }
  const size_t mm = (size_t)m * m;
  double *Y = (double *)malloc(sizeof(double) * (size_t)kdim * m);
  double *Hh = (double *)malloc(sizeof(double) * 2 * mm);
  double *Zh = (double *)malloc(sizeof(double) * mm);
  double *lam = (double *)malloc(sizeof(double) * (size_t)m);
  double *hv = (double *)malloc(sizeof(double) * (size_t)m);
  double *U = (double *)ws(WS_RITZ, sizeof(double) * (size_t)ld * m);
  double *P = (double *)ws(WS_RITZ2, sizeof(double) * (size_t)ld * m);
  double *W = (double *)ws(WS_REF1, sizeof(double) * (size_t)ld * m);
  double *X = (double *)ws(WS_REF2, sizeof(double) * (size_t)ld * m);
  void *fwork = ws(WS_FILT, 16 * (size_t)ld * kMaxBatch);
  double *dmu = (double *)ws(WS_MU, sizeof(double) * (size_t)(S->pol->deg + 1));
  if (dmu && memcpy_async(dmu, S->pol->mu, sizeof(double) * (size_t)(S->pol->deg + 1))) dmu = nullptr;
  /* small device matrices: Y | G | H | Z | 3 m scalars */
  double *dsm = (double *)ws(WS_H, sizeof(double) * ((size_t)kdim * m + 3 * mm + 3 * (size_t)m));
  if (!Y || !Hh || !Zh || !lam || !hv || !U || !P || !W || !X || !fwork || !dsm || !dmu)
    st = PEVSL_ERR_NOMEM;
  double *dY = dsm, *dG = dY + (size_t)kdim * m, *dH = dG + mm, *dZ = dH + mm, *dv = dZ + mm;
  if (!st && pevsl_tridiag_eig_sel(kdim, S->dT, S->eT, S->EvalT, m, sel, Y)) st = PEVSL_ERR_EIG;
  /* largest Ritz values first: the Cholesky of G then keeps the wanted
   * directions and drops guard columns that became dependent on them */
  for (int j = 0; j < m / 2 && !st; j++) {
    double *c1 = Y + (size_t)j * kdim, *c2 = Y + (size_t)(m - 1 - j) * kdim;
    for (int i = 0; i < kdim; i++) {
      const double t = c1[i];
      c1[i] = c2[i];
      c2[i] = t;
    }
  }
  /* U = V Y; P = p(A) U in FP64, unit columns */
  if (!st) st = memcpy_async(dY, Y, sizeof(double) * (size_t)kdim * m);
  if (!st) st = gemm_nn(n, kdim, m, S->V, ld, dY, kdim, U, ld);
  for (int pass = 0; pass < passes && !st; pass++) {
    double *src = pass % 2 == 0 ? U : P, *dst = pass % 2 == 0 ? P : U;
    for (int c0 = 0; c0 < m && !st; c0 += kMaxBatch) {
      const int cs = PEVSL_MIN(kMaxBatch, m - c0);
      FilterJob jobs[kMaxBatch];
      for (int e = 0; e < cs; e++)
        jobs[e] = FilterJob{pevsl, A, src + (size_t)(c0 + e) * ld, dst + (size_t)(c0 + e) * ld,
                            S->pol, dmu, (char *)fwork + 16 * (size_t)ld * e, ld};
      st = cheb_filter_batch(cs, jobs, false);
    }
    if (!st) st = vdot_cols(n, m, dst, ld, dst, ld, dv);
    if (!st) st = memcpy_async(hv, dv, sizeof(double) * m);
    if (!st) st = sync();
    for (int j = 0; j < m && !st; j++) hv[j] = hv[j] > 0 ? 1.0 / sqrt(hv[j]) : 0.0;
    if (!st) st = memcpy_async(dv, hv, sizeof(double) * m);
    if (!st) st = vscal_cols(n, m, dst, ld, dv);
  }
  if (!st && passes % 2 == 0) st = vcopy(U, P, (long)ld * m); /* filtered block in P */
  /* W = A P; G = P'P, H = P'W */
  for (int j = 0; j < m && !st; j++) st = spmv(A, P + (size_t)j * ld, W + (size_t)j * ld);
  pevsl->stats->n_mvA += (size_t)m;
  if (!st) st = gemm_tn(n, m, m, P, ld, P, ld, dG, m);
  if (!st) st = gemm_tn(n, m, m, P, ld, W, ld, dH, m);
  if (!st) st = memcpy_async(Hh, dG, sizeof(double) * 2 * mm);
  if (!st) st = sync();
  int q = 0;
  if (!st) {
    double *G = Hh, *H = Hh + mm;
    for (int i = 0; i < m; i++)
      for (int j = 0; j < i; j++) {
        const double g = 0.5 * (G[(size_t)j * m + i] + G[(size_t)i * m + j]);
        const double h = 0.5 * (H[(size_t)j * m + i] + H[(size_t)i * m + j]);
        G[(size_t)j * m + i] = G[(size_t)i * m + j] = g;
        H[(size_t)j * m + i] = H[(size_t)i * m + j] = h;
      }
    const double te = pevsl_now();
    st = pevsl_gen_symeig_range(m, H, G, m, aa - DBL_EPSILON, bb + DBL_EPSILON, &q, lam, Zh, m);
    pevsl->stats->t_eig += pevsl_now() - te;
  }
  pEVSL_ParvecsDuplParvec(vinit, q, (int)n, S->Rvec);
  if (!st && q > 0) {
    /* X = P Z, A X = W Z (into U), unit columns, R = A X - lam X */
    st = memcpy_async(dZ, Zh, sizeof(double) * (size_t)m * q);
    if (!st) st = gemm_nn(n, m, q, P, ld, dZ, m, X, ld);
    if (!st) st = gemm_nn(n, m, q, W, ld, dZ, m, U, ld);
    if (!st) st = vdot_cols(n, q, X, ld, X, ld, dv);
    if (!st) st = memcpy_async(hv, dv, sizeof(double) * q);
    if (!st) st = sync();
    for (int j = 0; j < q && !st; j++) hv[j] = hv[j] > 0 ? 1.0 / sqrt(hv[j]) : 0.0;
    if (!st) st = memcpy_async(dv, hv, sizeof(double) * q);
    if (!st) st = vscal_cols(n, q, X, ld, dv);
    if (!st) st = vscal_cols(n, q, U, ld, dv);
    if (!st) st = memcpy_async(dv + m, lam, sizeof(double) * q);
    if (!st) st = vaxpy_cols(n, q, dv + m, X, ld, U, ld);
    if (!st) st = vdot_cols(n, q, U, ld, U, ld, dv + 2 * m);
    if (!st) st = memcpy_async(hv, dv + 2 * m, sizeof(double) * q);
    if (!st) st = sync();
    double rmin = HUGE_VAL, rmax = 0.0;
    for (int j = 0; j < q && !st; j++) {
      const double r0 = sqrt(hv[j]);
      rmin = PEVSL_MIN(rmin, r0);
      rmax = PEVSL_MAX(rmax, r0);
      if (r0 < tol) {
        S->Lam[S->nev] = lam[j];
        S->res[S->nev] = r0;
        st = vcopy(X + (size_t)j * ld, S->Rvec->data + (size_t)S->nev * S->Rvec->ld, n);
        S->nev++;
      }
    }
    if (!st) st = sync();
    /* a refined pair in [a, b] short of the FP64 path's quality (residual
     * below tol, and below tol * |lam| for |lam| < 1) sends the slice back
     * to FP64 */
    int weak = 0;
    for (int j = 0; j < q; j++)
      if (!(sqrt(hv[j]) < tol * PEVSL_MIN(1.0, fabs(lam[j])))) weak++;
    S->short_pairs = PEVSL_MAX(weak, nbar - S->nev);
    if (getenv("PEVSL_B200_VERBOSE"))
      fprintf(stderr, "refine [%g, %g]: kdim %d, subspace %d, in [a,b] %d, accepted %d, res %.2e..%.2e\n",
              aa, bb, kdim, m, q, S->nev, rmin, rmax);
  } else if (getenv("PEVSL_B200_VERBOSE")) {
    fprintf(stderr, "refine [%g, %g]: kdim %d, subspace %d, in [a,b] %d, status %d\n", aa, bb, kdim,
            m, q, st);
  }
  free(sel);
  free(Y);
  free(Hh);
  free(Zh);
  free(lam);
  free(hv);
  return st;
}

static void free_slice_outputs(SliceState *S) {
  free(S->Lam);
  free(S->res);
  if (S->Rvec) {
    pEVSL_ParvecsFree(S->Rvec);
    free(S->Rvec);
  }
  S->Lam = S->res = nullptr;
  S->Rvec = nullptr;
}

/* Lockstep filtered Lanczos over ns <= kMaxBatch slices sharing vinit. */
static int g_fallbacks = 0; /* slices of the last call re-run in FP64 */

int pEVSL_B200_LastFallbacks(void) { return g_fallbacks; }

int pEVSL_B200_SetGroupReduce(pevsl_Data *pevsl, void (*reduce)(double *buf, int count, void *ctx),
                              void *ctx) {
  if (!pevsl) return PEVSL_ERR_ARG;
  pevsl_inst *inst = pevsl_inst_of(pevsl);
  inst->group_reduce = reduce;
  inst->group_reduce_ctx = ctx;
  return 0;
}

int pEVSL_B200_SetFilterForm(int form) {
  if (form < -1 || form > 2) return PEVSL_ERR_ARG;
  g_filter_form_override = form < 0 ? 2 : form;
  return 0;
}

int pEVSL_B200_SetBarrierSpins(unsigned spins) {
  set_barrier_spins(spins);
  return 0;
}

int pEVSL_B200_SeedBarrierArrivals(unsigned count) { return seed_barrier_arrivals(count); }

int pEVSL_B200_SetClusterWait(long microseconds) {
  set_cluster_wait(microseconds);
  return 0;
}

int pEVSL_B200_WithholdClusterValues(int on) {
  withhold_cluster_values(on != 0);
  return 0;
}

/* Filtered Lanczos in lockstep (pEVSL_ChebLanNr, SRC/cheblanNr.c:54-448) for
 * ns <= kMaxEntries slices, which may belong to different problems (each
 * entry carries its instance, matrix, length and start vector).  Every
 * step runs one filter application for all active slices (one launch per
 * degree, or one persistent launch), then the Lanczos recurrence and
 * CGS-DGKS as batched launches of up to kMaxBatch entries.  Per entry the
 * work decomposition is that of a one-slice run, so each slice's result is
 * bit-identical to solving it alone. */
static int cheblannr_group(SliceState *SL, int ns, double tol, FILE *fstats,
                           bool allow_mixed = true) {
  Ctx &c = ctx();
  if (ns <= 0) return 0;
  if (ns > kMaxEntries) return PEVSL_ERR_ARG;
  const bool mixed = allow_mixed && SL[0].A &&
                     pevsl_inst_of(SL[0].pevsl)->precision == PEVSL_PREC_MIXED;
  bool all_builtin = true;
  long nmax = 0;
  for (int s = 0; s < ns; s++) {
    all_builtin = all_builtin && SL[s].A != nullptr;
    nmax = PEVSL_MAX(nmax, SL[s].n);
  }
  /* the lockstep machinery also serves one slice when the filter is
   * graph-replayed (one captured launch sequence per filter application) */
  const bool batched = all_builtin && (ns > 1 || mixed || filter_graph_enabled());
  /* mixed form: trace tolerance per converged value, and the guard of the
   * refinement sweep (PEVSL_B200_MIXED_TRTOL / PEVSL_B200_MIXED_GUARD) */
  double trtol_mixed = 1e-9, guard = 0.3;
  int passes = 1;
  if (getenv("PEVSL_B200_MIXED_TRTOL")) trtol_mixed = atof(getenv("PEVSL_B200_MIXED_TRTOL"));
  if (getenv("PEVSL_B200_MIXED_GUARD")) guard = atof(getenv("PEVSL_B200_MIXED_GUARD"));
  if (getenv("PEVSL_B200_MIXED_PASSES")) passes = PEVSL_MAX(1, atoi(getenv("PEVSL_B200_MIXED_PASSES")));
  std::vector<char> act(ns, 0);
  int nact = 0;
  size_t basis_elems = 0, work_bytes = 0, mu_elems = 0;
  for (int s = 0; s < ns; s++) {
    SliceState *S = &SL[s];
    S->maxit = PEVSL_MIN(S->pevsl->N, S->maxit);
    S->status = 0;
    S->nev = 0;
    S->its = 0;
    S->short_pairs = 0;
    if (pevsl_check_intv(S->intv, fstats) < 0) {
      S->done = 1; /* invalid interval: no pairs, status 0 (SRC/cheblanNr.c:96-100) */
      continue;
    }
    if (fstats) {
      fprintf(fstats, " intv:[%e, %e, %e, %e]\n", S->intv[0], S->intv[1], S->intv[2], S->intv[3]);
      fprintf(fstats, " ** Cheb Poly of deg = %d, gam = %.15e, bar: %.15e\n", S->pol->deg,
              S->pol->gam, S->pol->bar);
    }
    if (S->pol->gam > 1.0 || S->pol->gam < -1.0) {
      fprintf(stdout, "gamB error %.15e\n", S->pol->gam);
      S->status = -1;
      S->done = 1;
      continue;
    }
    if (fstats) fprintf(fstats, " ** Cheb-LanNr \n");
    act[s] = 1;
    nact++;
    basis_elems += (size_t)S->ld * ((size_t)S->maxit + 1);
    work_bytes += 32 * (size_t)S->ld; /* filter work + the graph form's staging */
    mu_elems += (size_t)S->pol->deg + 1;
  }
  if (!nact) return 0;
  /* tune each matrix's stream kernels now: the filter may be captured */
  for (int s = 0; s < ns; s++)
    if (act[s] && SL[s].A && stream_tune(SL[s].A)) return PEVSL_ERR_CUDA;
  if (mixed)
    for (int s = 0; s < ns; s++)
      if (act[s] && csr_make_fp32(SL[s].A)) return PEVSL_ERR_NOMEM;
  /* bases of all active slices in one workspace; three FP64 vectors for
   * the one-slice filter and breakdown restarts; 16 ld bytes of batched
   * filter work per slice; the filter coefficients on the device */
  double *Vall = (double *)ws(WS_BASIS, sizeof(double) * basis_elems);
  const size_t w3len = (size_t)round_ld(3 * nmax);
  double *w3 = (double *)ws(WS_CHEB, sizeof(double) * w3len + (batched ? work_bytes : 0));
  double *vrand = (double *)ws(all_builtin ? WS_VEC : WS_RITZ2, sizeof(double) * (size_t)nmax);
  double *dmu_all = batched ? (double *)ws(WS_MU, sizeof(double) * mu_elems) : nullptr;
  if (!Vall || !w3 || !vrand || (batched && !dmu_all)) return PEVSL_ERR_NOMEM;
  char *bwork = (char *)(w3 + w3len);
  std::vector<char *> work(ns, nullptr);
  std::vector<const double *> dmu(ns, nullptr);
  int st = 0;
  size_t off = 0, woff = 0, moff = 0;
  int maxit_all = 0;
  for (int s = 0; s < ns && !st; s++) {
    SliceState *S = &SL[s];
    if (!act[s]) continue;
    S->V = Vall + off;
    off += (size_t)S->ld * ((size_t)S->maxit + 1);
    if (batched) {
      work[s] = bwork + woff;
      woff += 32 * (size_t)S->ld;
      dmu[s] = dmu_all + moff;
      st = memcpy_async(dmu_all + moff, S->pol->mu, sizeof(double) * ((size_t)S->pol->deg + 1));
      moff += (size_t)S->pol->deg + 1;
    }
    S->dT = (double *)malloc(sizeof(double) * (size_t)S->maxit);
    S->eT = (double *)malloc(sizeof(double) * (size_t)S->maxit);
    S->EvalT = (double *)malloc(sizeof(double) * (size_t)S->maxit);
    if (!S->dT || !S->eT || !S->EvalT) return PEVSL_ERR_NOMEM;
    S->wn = S->tr0 = S->beta = 0.0;
    S->nwn = S->kdim = S->count = S->nconv = 0;
    maxit_all = PEVSL_MAX(maxit_all, S->maxit);
  }
  if (st) return st;
  SegTimer &t_pol = g_t_pol, &t_orth = g_t_orth;
  /* CUDA graph form of the batched filter: one captured launch sequence per
   * set of live slices, replayed every step */
  const bool graph_form = batched && filter_form() == 0 && filter_graph_enabled();
  FilterGraph fg;
  fg.mixed = mixed;
  /* y_s = p_s(A_s) x_s for the slices with sel[s]: x_s = V_s(:,kin) (or the
   * slice's start vector when xin), y_s = V_s(:,kout) */
  auto filter = [&](const std::vector<char> &sel, int kin, bool xin, int kout) -> int {
    t_pol.begin();
    int r = 0;
    if (!batched) {
      for (int s = 0; s < ns && !r; s++)
        if (sel[s])
          r = cheb_apply(SL[s].pevsl, SL[s].pol,
                         xin ? SL[s].vinit->data : SL[s].V + (size_t)kin * SL[s].ld,
                         SL[s].V + (size_t)kout * SL[s].ld, w3, SL[s].n);
    } else {
      std::vector<FilterJob> jobs;
      jobs.reserve(ns);
      for (int s = 0; s < ns; s++)
        if (sel[s])
          jobs.push_back(FilterJob{SL[s].pevsl, SL[s].A,
                                   xin ? SL[s].vinit->data : SL[s].V + (size_t)kin * SL[s].ld,
                                   SL[s].V + (size_t)kout * SL[s].ld, SL[s].pol, dmu[s], work[s],
                                   SL[s].ld});
      /* with every application one cluster launch there is nothing to capture */
      if (graph_form && !all_cluster(jobs, mixed))
        r = filter_graphed(fg, sel, jobs);
      else
        r = cheb_filter_batch((int)jobs.size(), jobs.data(), mixed);
    }
    t_pol.end();
    return r;
  };
  /* a batched operation over the active entries, kMaxBatch at a time:
   * op(first entry, count, mask, lengths) */
  auto chunks = [&](const std::vector<char> &sel, auto &&op) -> int {
    for (int c0 = 0; c0 < ns; c0 += kMaxBatch) {
      const int cs = PEVSL_MIN(kMaxBatch, ns - c0);
      unsigned mask = 0;
      BLen len{};
      for (int i = 0; i < cs; i++) {
        len.n[i] = SL[c0 + i].n;
        len.ld[i] = SL[c0 + i].ld;
        if (sel[c0 + i]) mask |= 1u << i;
      }
      if (!mask) continue;
      const int r = op(c0, cs, mask, len);
      if (r) return r;
    }
    return 0;
  };
  /* per-entry device scalars: alpha, ||v|| before CGS, ||v|| after, and the
   * DGKS flag */
  double *dA = c.gscal, *dN0 = c.gscal + kMaxEntries, *dN = c.gscal + 2 * kMaxEntries;
  double *hA = c.hgscal, *hN = c.hgscal + 2 * kMaxEntries;
  int *dF = c.gflag;
  const long ldw = maxit_all + 1;
  double *dW = (double *)ws(WS_GROUP, sizeof(double) * (size_t)ns * (size_t)ldw);
  if (!dW) return PEVSL_ERR_NOMEM;
  for (int s = 0; s < ns; s++)
    if (act[s] && SL[s].A) matrix_window(SL[s].A);
  cudaEvent_t e_all0, e_all1;
  cudaEventCreate(&e_all0);
  cudaEventCreate(&e_all1);
  cudaEventRecord(e_all0, c.stream);
  /* filter the start vector, normalise (SRC/cheblanNr.c:164-194) */
  st = filter(act, 0, true, 0);
  if (!st)
    st = chunks(act, [&](int c0, int cs, unsigned mask, const BLen &len) {
      CPtrs x{};
      for (int i = 0; i < cs; i++) x.p[i] = SL[c0 + i].V;
      return b_dot(len, cs, x, x, dA + c0, FIN_SQRT, mask);
    });
  if (!st) st = memcpy_async(hA, dA, sizeof(double) * (size_t)ns);
  if (!st) st = sync();
  if (!st)
    st = chunks(act, [&](int c0, int cs, unsigned mask, const BLen &len) {
      BScal inv{};
      VPtrs y{};
      for (int i = 0; i < cs; i++) {
        inv.v[i] = 1.0 / hA[c0 + i];
        y.p[i] = SL[c0 + i].V;
      }
      return b_scal(len, cs, y, inv, mask);
    });
  int k;
  for (k = 0; nact > 0 && !st; k++) {
    st = filter(act, k, false, k + 1);
    auto col = [&](int s, int j) { return SL[s].V + (size_t)j * SL[s].ld; };
    if (!st && k > 0)
      st = chunks(act, [&](int c0, int cs, unsigned mask, const BLen &len) {
        CPtrs vprev{};
        VPtrs vnew{};
        BScal mb{};
        for (int i = 0; i < cs; i++) {
          vprev.p[i] = col(c0 + i, k - 1);
          vnew.p[i] = col(c0 + i, k + 1);
          mb.v[i] = -SL[c0 + i].beta;
        }
        return b_axpy(len, cs, vprev, vnew, mb, mask);
      });
    if (!st)
      st = chunks(act, [&](int c0, int cs, unsigned mask, const BLen &len) {
        CPtrs vk{}, vks{};
        for (int i = 0; i < cs; i++) {
          vk.p[i] = col(c0 + i, k);
          vks.p[i] = col(c0 + i, k + 1);
        }
        return b_dot(len, cs, vk, vks, dA + c0, FIN_ID, mask);
      });
    t_orth.begin();
    /* v -= alpha v_k, ||v||; CGS_DGKS: pass 1, then pass 2 where the first
     * kept <= 1/sqrt(2) of the norm */
    if (!st)
      st = chunks(act, [&](int c0, int cs, unsigned mask, const BLen &len) {
        CPtrs vk{}, Vc{}, vks{};
        VPtrs vnew{};
        for (int i = 0; i < cs; i++) {
          vk.p[i] = col(c0 + i, k);
          vnew.p[i] = col(c0 + i, k + 1);
          vks.p[i] = vnew.p[i];
          Vc.p[i] = SL[c0 + i].V;
        }
        int r = b_axpy_dev_nrm2(len, cs, dA + c0, vk, vnew, dN0 + c0, mask);
        double *w = dW + (size_t)c0 * ldw;
        if (!r) r = b_gemvT(len, cs, k + 1, Vc, vks, w, ldw, nullptr, mask);
        if (!r)
          r = b_gemv_sub_nrm(len, cs, k + 1, Vc, w, ldw, vnew, dN + c0, nullptr, dF + c0, dN0 + c0,
                             kEta, mask);
        if (!r) r = b_gemvT(len, cs, k + 1, Vc, vks, w, ldw, dF + c0, mask);
        if (!r)
          r = b_gemv_sub_nrm(len, cs, k + 1, Vc, w, ldw, vnew, dN + c0, dF + c0, nullptr, nullptr,
                             kEta, mask);
        return r;
      });
    t_orth.end();
    if (!st) st = memcpy_async(hA, dA, sizeof(double) * (size_t)ns);
    if (!st) st = memcpy_async(hN, dN, sizeof(double) * (size_t)ns);
    if (!st) st = sync();
    if (st) break;
    t_pol.flush();
    t_orth.flush();
    std::vector<char> scal_sel(ns, 0);
    std::vector<double> inv(ns, 0.0);
    for (int s = 0; s < ns && !st; s++) {
      if (!act[s]) continue;
      SliceState *S = &SL[s];
      const double alpha = hA[s];
      double beta = hN[s];
      if (!isfinite(alpha) || !isfinite(beta)) {
        S->status = PEVSL_ERR_NONFINITE;
        S->done = 1;
        act[s] = 0;
        nact--;
        continue;
      }
      S->dT[k] = alpha;
      S->wn += fabs(alpha);
      S->wn += 2.0 * beta;
      S->nwn += 3;
      double *znew = S->V + (size_t)(k + 1) * S->ld;
      if (beta * S->nwn < orthTol * S->wn) {
        /* lucky breakdown: restart from a new filtered random vector
         * (SRC/cheblanNr.c:248-281) */
        if (fstats) fprintf(fstats, "it %4d: Lucky breakdown, beta = %.15e\n", k, beta);
        st = pevsl_rand_vector_dev(vrand, (int)S->n);
        t_pol.begin();
        if (!st) st = cheb_apply(S->pevsl, S->pol, vrand, znew, w3, S->n);
        t_pol.end();
        if (!st) st = vnrm2(S->n, znew, c.dscal + S_NRM0);
        if (!st) st = cgs_dgks(S->V, S->ld, k + 1, znew, S->n);
        const double *hb = st ? nullptr : fetch_scalars(S_NRM, 1);
        if (!hb) {
          st = st ? st : PEVSL_ERR_CUDA;
          break;
        }
        st = vscal(znew, S->n, 1.0 / hb[0]);
        beta = 0.0;
      } else {
        inv[s] = 1.0 / beta;
        scal_sel[s] = 1;
      }
      S->beta = beta;
      S->eT[k] = beta;
    }
    if (!st)
      st = chunks(scal_sel, [&](int c0, int cs, unsigned mask, const BLen &len) {
        BScal v{};
        VPtrs sc{};
        for (int i = 0; i < cs; i++) {
          v.v[i] = inv[c0 + i];
          sc.p[i] = col(c0 + i, k + 1);
        }
        return b_scal(len, cs, sc, v, mask);
      });
    if (st) break;
    /* restricted-trace convergence test (SRC/cheblanNr.c:293-332); the
     * eigenvalues of the testing slices' T are computed first, on host
     * threads (each slice's own arithmetic, so the same values), then the
     * tests run in slice order */
    std::vector<int> tests;
    for (int s = 0; s < ns; s++)
      if (act[s] && !((k < 30 || (k - 30) % 20 != 0) && k != SL[s].maxit - 1)) tests.push_back(s);
    std::vector<int> eig_st(tests.size(), 0);
    std::vector<double> eig_secs(tests.size(), 0.0);
    host_parallel(tests.size(), k + 1 >= 64, [&](size_t i) {
      SliceState *S = &SL[tests[i]];
      const double te = pevsl_now();
      eig_st[i] = pevsl_tridiag_eig(k + 1, S->dT, S->eT, S->EvalT, nullptr);
      eig_secs[i] = pevsl_now() - te;
    });
    for (size_t ti = 0; ti < tests.size(); ti++) {
      const int s = tests[ti];
      SliceState *S = &SL[s];
      S->kdim = k + 1;
      if (eig_st[ti]) {
        st = PEVSL_ERR_EIG;
        break;
      }
      S->pevsl->stats->t_eig += eig_secs[ti];
      S->count = S->kdim;
      double tr1 = 0.0;
      S->nconv = 0;
      for (int i = 0; i < S->count; i++) {
        if (S->EvalT[i] + 5 * DBL_EPSILON >= S->pol->bar) {
          tr1 += S->EvalT[i];
          S->nconv++;
        }
      }
      if (fstats) fprintf(fstats, "  k %4d:   nconv %4d  tr1 %21.15e\n", k, S->nconv, tr1);
      /* FP64: the reference's test; mixed: differences at the FP32 noise
       * level of the filtered operator count as converged */
      const double trtol = mixed ? trtol_mixed * PEVSL_MAX(1, S->nconv) : 2e-12;
      const bool conv = fabs(tr1 - S->tr0) < trtol || fabs(tr1) + fabs(S->tr0) < 1e-10;
      S->tr0 = tr1;
      if (conv || k == S->maxit - 1) {
        if (!conv && fstats)
          fprintf(fstats, "The max number of iterations [%d] has been reached. The eigenvalues "
                          "computed may not have converged\n", S->maxit);
        act[s] = 0;
        nact--;
      }
    }
  }
  cudaEventRecord(e_all1, c.stream);
  const double tr_start = pevsl_now();
  /* the host part of every finished slice's Ritz extraction first, on host
   * threads; then the device part slice by slice */
  std::vector<RitzHost> rh((size_t)ns);
  if (!st && !mixed) {
    std::vector<int> fin;
    int kmax = 0;
    for (int s = 0; s < ns; s++)
      if (!SL[s].done && !SL[s].status) {
        fin.push_back(s);
        kmax = PEVSL_MAX(kmax, SL[s].kdim);
      }
    host_parallel(fin.size(), kmax >= 64, [&](size_t i) { ritz_host(&SL[fin[i]], &rh[fin[i]]); });
  }
  for (int s = 0; s < ns && !st; s++) {
    SliceState *S = &SL[s];
    if (S->done || S->status) continue;
    S->its = S->kdim;
    const int rs = mixed ? ritz_refine(S->pevsl, S, S->vinit, S->n, S->ld, tol, guard, passes)
                         : ritz_extract(S->pevsl, S, &rh[s], S->vinit, S->n, S->ld, tol);
    if (rs) S->status = rs;
  }
  for (RitzHost &R : rh) {
    free(R.sel);
    free(R.Y);
  }
  for (int s = 0; s < ns; s++) SL[s].pevsl->stats->t_ritz = pevsl_now() - tr_start;
  cudaEventSynchronize(e_all1);
  t_pol.flush();
  t_orth.flush();
  float ms_all = 0.f;
  cudaEventElapsedTime(&ms_all, e_all0, e_all1);
  cudaEventDestroy(e_all0);
  cudaEventDestroy(e_all1);
  for (int s = 0; s < ns; s++) {
    pevsl_inst *inst = pevsl_inst_of(SL[s].pevsl);
    if (s > 0 && SL[s].pevsl == SL[s - 1].pevsl) continue;
    inst->phase_ms[2] = ms_all;
    inst->phase_ms[3] = t_pol.acc_ms;
    inst->phase_ms[4] = t_orth.acc_ms;
    SL[s].pevsl->stats->t_polAv += 1e-3 * t_pol.acc_ms;
    SL[s].pevsl->stats->t_reorth += 1e-3 * t_orth.acc_ms;
  }
  if (all_builtin) g_filter_ms += t_pol.acc_ms;
  for (int s = 0; s < ns; s++) {
    free(SL[s].dT);
    free(SL[s].eT);
    free(SL[s].EvalT);
    SL[s].dT = SL[s].eT = SL[s].EvalT = nullptr;
  }
  if (mixed && !st) {
    /* a slice is run again in FP64 when a refined pair in [a, b] misses the
     * FP64 path's quality, or fewer pairs were accepted than the Lanczos
     * run had Ritz values above bar, so the mixed form never reports fewer
     * or worse pairs */
    std::vector<SliceState> R;
    std::vector<int> idx;
    for (int s = 0; s < ns; s++) {
      SliceState *S = &SL[s];
      if (S->done || S->status || S->short_pairs <= 0) continue;
      free_slice_outputs(S);
      SliceState r;
      memset(&r, 0, sizeof r);
      memcpy(r.intv, S->intv, sizeof S->intv);
      r.pol = S->pol;
      r.maxit = S->maxit;
      r.pevsl = S->pevsl;
      r.A = S->A;
      r.vinit = S->vinit;
      r.n = S->n;
      r.ld = S->ld;
      R.push_back(r);
      idx.push_back(s);
    }
    if (!R.empty()) {
      g_fallbacks += (int)R.size();
      pevsl_inst *inst = pevsl_inst_of(SL[0].pevsl);
      const float ms0 = inst->phase_ms[2], pol0 = inst->phase_ms[3], orth0 = inst->phase_ms[4];
      st = cheblannr_group(R.data(), (int)R.size(), tol, fstats, false);
      inst->phase_ms[2] += ms0;
      inst->phase_ms[3] += pol0;
      inst->phase_ms[4] += orth0;
      for (size_t r = 0; r < R.size(); r++) {
        SliceState *S = &SL[idx[r]];
        S->status = R[r].status;
        S->kdim = R[r].kdim;
        S->its = R[r].its;
        S->nconv = R[r].nconv;
        S->nev = R[r].nev;
        S->Lam = R[r].Lam;
        S->res = R[r].res;
        S->Rvec = R[r].Rvec;
        S->short_pairs = 0;
      }
    }
  }
  return st;
}

static void slice_bind(SliceState *S, pevsl_Data *pevsl, pevsl_Parvec *vinit) {
  S->pevsl = pevsl;
  S->A = pevsl_builtin_A(pevsl);
  S->vinit = vinit;
  S->n = pevsl->n;
  S->ld = round_ld(pevsl->n);
}

int pEVSL_ChebLanNr(pevsl_Data *pevsl, double *intv, int maxit, double tol, pevsl_Parvec *vinit,
                    pevsl_Polparams *pol, int *nevOut, double **lamo, pevsl_Parvecs **Wo,
                    double **reso, FILE *fstats) {
  const double tall = pevsl_now();
  *nevOut = 0;
  *lamo = nullptr;
  *Wo = nullptr;
  *reso = nullptr;
  if (ensure()) return PEVSL_ERR_CUDA;
  if (pevsl->ifGenEv) {
    int its = 0;
    const int st = pevsl_gen_cheblannr(pevsl, intv, maxit, tol, vinit, pol, nevOut, lamo, Wo, reso,
                                       &its, fstats);
    pevsl_inst_of(pevsl)->last_its = its;
    pevsl->stats->t_iter = pevsl_now() - tall;
    return st;
  }
  SliceState S;
  memset(&S, 0, sizeof S);
  memcpy(S.intv, intv, sizeof S.intv);
  S.pol = pol;
  S.maxit = maxit;
  slice_bind(&S, pevsl, vinit);
  g_t_pol.init();
  g_t_orth.init();
  g_fallbacks = 0;
  int st = cheblannr_group(&S, 1, tol, fstats);
  pevsl_inst *inst = pevsl_inst_of(pevsl);
  inst->last_its = S.kdim;
  inst->last_nconv = S.nconv;
  if (!st) st = S.status;
  if (st) {
    free_slice_outputs(&S);
    return st;
  }
  *nevOut = S.nev;
  *lamo = S.Lam;
  *Wo = S.Rvec;
  *reso = S.res;
  pevsl->stats->t_iter = pevsl_now() - tall;
  return 0;
}

/* outputs of a solved group into the caller's arrays at offset o */
static int group_outputs(SliceState *SL, int ns, int st, int o, int *nevOut, double **lamo,
                         pevsl_Parvecs **Wo, double **reso, int *its, int *status) {
  int first_err = 0;
  for (int s = 0; s < ns; s++) {
    SliceState *S = &SL[s];
    const int ss = st ? st : S->status;
    status[o + s] = ss;
    its[o + s] = S->kdim;
    if (ss) {
      free_slice_outputs(S);
      nevOut[o + s] = 0;
      lamo[o + s] = nullptr;
      Wo[o + s] = nullptr;
      reso[o + s] = nullptr;
      if (!first_err) first_err = ss;
    } else {
      nevOut[o + s] = S->nev;
      lamo[o + s] = S->Lam;
      Wo[o + s] = S->Rvec;
      reso[o + s] = S->res;
    }
  }
  return first_err;
}

int pEVSL_B200_ChebLanNrBatch(pevsl_Data *pevsl, int nslices, const double *intvs,
                              const int *maxits, double tol, pevsl_Parvec *vinit,
                              pevsl_Polparams *pols, int *nevOut, double **lamo,
                              pevsl_Parvecs **Wo, double **reso, int *its, int *status,
                              FILE *fstats) {
  const double tall = pevsl_now();
  if (ensure()) return PEVSL_ERR_CUDA;
  if (nslices < 0) return PEVSL_ERR_ARG;
  int first_err = 0;
  if (pevsl->ifGenEv) {
    /* generalized problem: in lockstep where the lockstep form applies,
     * else the slices one after the other */
    if (nslices >= 2 && nslices <= kMaxBatch) {
      const int r = pevsl_gen_cheblannr_lockstep(pevsl, nslices, intvs, maxits, tol, vinit, pols,
                                                 nevOut, lamo, Wo, reso, its, status, fstats);
      if (r != 1) {
        pevsl->stats->t_iter = pevsl_now() - tall;
        return r;
      }
    }
    for (int s = 0; s < nslices; s++) {
      double iv[4];
      memcpy(iv, intvs + 4 * (size_t)s, sizeof iv);
      status[s] = pevsl_gen_cheblannr(pevsl, iv, maxits[s], tol, vinit, &pols[s], &nevOut[s],
                                      &lamo[s], &Wo[s], &reso[s], &its[s], fstats);
      if (status[s] && !first_err) first_err = status[s];
    }
    pevsl->stats->t_iter = pevsl_now() - tall;
    return first_err;
  }
  g_t_pol.init();
  g_t_orth.init();
  g_fallbacks = 0;
  double ms_total = 0.0, pol_total = 0.0, orth_total = 0.0;
  for (int s0 = 0; s0 < nslices; s0 += kMaxEntries) {
    const int ns = PEVSL_MIN(kMaxEntries, nslices - s0);
    std::vector<SliceState> SL(ns);
    memset(SL.data(), 0, sizeof(SliceState) * (size_t)ns);
    for (int s = 0; s < ns; s++) {
      memcpy(SL[s].intv, intvs + 4 * (size_t)(s0 + s), sizeof SL[s].intv);
      SL[s].pol = &pols[s0 + s];
      SL[s].maxit = maxits[s0 + s];
      slice_bind(&SL[s], pevsl, vinit);
    }
    int st = cheblannr_group(SL.data(), ns, tol, fstats);
    pevsl_inst *inst = pevsl_inst_of(pevsl);
    ms_total += inst->phase_ms[2];
    pol_total += inst->phase_ms[3];
    orth_total += inst->phase_ms[4];
    const int e = group_outputs(SL.data(), ns, st, s0, nevOut, lamo, Wo, reso, its, status);
    if (!first_err) first_err = e;
  }
  pevsl_inst *inst = pevsl_inst_of(pevsl);
  inst->phase_ms[2] = ms_total;
  inst->phase_ms[3] = pol_total;
  inst->phase_ms[4] = orth_total;
  pevsl->stats->t_iter = pevsl_now() - tall;
  return first_err;
}

int pEVSL_B200_ChebLanNrMulti(int nprob, pevsl_Data **pevsls, const int *nslices,
                              const double *intvs, const int *maxits, double tol,
                              pevsl_Parvec **vinits, pevsl_Polparams *pols, int *nevOut,
                              double **lamo, pevsl_Parvecs **Wo, double **reso, int *its,
                              int *status, FILE *fstats) {
  if (ensure()) return PEVSL_ERR_CUDA;
  if (nprob < 0 || (nprob > 0 && (!pevsls || !nslices || !vinits))) return PEVSL_ERR_ARG;
  for (int p = 0; p < nprob; p++) {
    if (!pevsls[p] || nslices[p] < 0) return PEVSL_ERR_ARG;
  }
  g_t_pol.init();
  g_t_orth.init();
  g_fallbacks = 0;
  int first_err = 0;
  /* groups of up to kMaxEntries slices; a problem is kept in one group
   * where it fits, a problem with more slices fills groups of its own */
  std::vector<SliceState> SL;
  int o = 0, o0 = 0;
  auto flush = [&]() {
    if (SL.empty()) return;
    const int st = cheblannr_group(SL.data(), (int)SL.size(), tol, fstats);
    const int e = group_outputs(SL.data(), (int)SL.size(), st, o0, nevOut, lamo, Wo, reso, its,
                                status);
    if (!first_err) first_err = e;
    o0 += (int)SL.size();
    SL.clear();
  };
  for (int p = 0; p < nprob; p++) {
    if (pevsls[p]->ifGenEv) {
      /* a generalized problem: its slices one after the other */
      flush();
      for (int s = 0; s < nslices[p]; s++, o++) {
        double iv[4];
        memcpy(iv, intvs + 4 * (size_t)o, sizeof iv);
        status[o] = pevsl_gen_cheblannr(pevsls[p], iv, maxits[o], tol, vinits[p], &pols[o],
                                        &nevOut[o], &lamo[o], &Wo[o], &reso[o], &its[o], fstats);
        if (status[o] && !first_err) first_err = status[o];
      }
      o0 = o;
      continue;
    }
    if (!SL.empty() && (int)SL.size() + nslices[p] > kMaxEntries) flush();
    for (int s = 0; s < nslices[p]; s++, o++) {
      if ((int)SL.size() == kMaxEntries) flush();
      SliceState S;
      memset(&S, 0, sizeof S);
      memcpy(S.intv, intvs + 4 * (size_t)o, sizeof S.intv);
      S.pol = &pols[o];
      S.maxit = maxits[o];
      slice_bind(&S, pevsls[p], vinits[p]);
      SL.push_back(S);
    }
  }
  flush();
  return first_err;
}

}  // extern "C"
