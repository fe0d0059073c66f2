"""The work whose speed is watched: the slicing path and its parts through the
public entry points, over the sizes they are used at.

listed() names twelve cases, draw(rng) makes more of the same ranges.  For
each, prepare(case, seed) builds what a program holds before the call (the
matrix on the GPU, the instance, filters, start vectors), run(state) is the
call, work(case) the bytes and operations it cannot do without, and
exact(case, seed) its result in 64-bit torch or numpy.

    import random
    from perf import cases
    for c in cases.listed():
        out = cases.run(cases.prepare(c, 1))

Eigenvalues are returned, residuals are not: a residual near 1e-9 is the
rounding of the run that made it.
"""
import ctypes as C
import math

import numpy as np
import torch

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

DEV = "cuda"


# ---------------------------------------------------------------- cases
def listed():
    return [
        # one filter application pEVSL_ChebAv on a grid of the README's size:
        # every degree is a few microseconds, launches and latency count
        dict(name="filter_grid20", kind="filter", matrix="grid", grid="19x20x21", deg=100, lo=0.05, hi=0.10),
        # the same at the benchmark's 10^6 rows, sides that divide nothing
        dict(name="filter_grid100", kind="filter", matrix="grid", grid="99x100x101", deg=300, lo=0.066, hi=0.068),
        # a general sparse matrix (about 17 entries per row scattered over a
        # band of +-5000, every value different): nothing to compress
        dict(name="filter_sparse", kind="filter", matrix="random", n=1000003, half=8, band=5000, deg=60,
             lo=0.48, hi=0.52),
        # KPM density of states at the benchmark's size and settings
        dict(name="dos_grid100", kind="dos", grid="101x100x99", mdeg=300, nvec=30),
        # Lanczos density of states, the other DOS of the drivers
        dict(name="landos_grid41", kind="landos", grid="41x43x40", msteps=40, nvec=20, npts=200),
        # thick-restart Lanczos bounds, the first step of every run
        dict(name="bounds_grid100", kind="bounds", grid="100x99x101", lanm=50, maxit=200),
        # the README run: KPM, slicing, filters and five slices in lockstep
        dict(name="run_grid20", kind="run", grid="20x21x19", first=60, count=120, slices=5, nvec=60, mdeg=300,
             mixed=False),
        # a smaller one with the FP32 filter and moments
        dict(name="run_grid16_mixed", kind="run", grid="17x15x16", first=40, count=60, slices=3, nvec=30,
             mdeg=200, mixed=True),
        # the drop-in call: one slice through pEVSL_ChebLanNr
        dict(name="slice_grid64", kind="slice", grid="65x64x63", first=80, count=20),
        # many problems at once: 2D and 3D grids of uneven size in lockstep
        dict(name="slices_multi", kind="multi", grids="59x61x60,181x179x1,28x27x29", first=40, count=14,
             slices=3),
        # a generalized problem A x = lambda B x, B a mass matrix with the
        # least-squares polynomial for B^{-1}, two slices in lockstep
        dict(name="gen_grid20", kind="gen", grid="20x19x21", first=30, count=8, slices=2),
        # the learned density of states: eight training steps (BF16 products,
        # forward and backward) and the prediction of a validation batch
        dict(name="learned_dos", kind="learned", moments=300, width=256, layers=4, batch=128, steps=8),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _sides(rng, n, dims=3):
    """Distinct sides near n^(1/dims), so that eigenvalues are simple."""
    s = max(6, int(round(n ** (1.0 / dims))))
    d = rng.sample(range(-max(2, s // 10), max(2, s // 10) + 1), dims)
    return "x".join(str(s + e) for e in d) + ("" if dims == 3 else "x1")


def draw(rng):
    kind = rng.choice(["filter", "filter", "random", "dos", "landos", "bounds", "run", "mixed", "slice", "multi",
                       "gen", "learned"])
    if kind == "filter":
        n = _log(rng, 4000, 1000000)
        lo = rng.uniform(0.02, 0.9)
        return dict(kind="filter", matrix="grid", grid=_sides(rng, n, rng.choice([2, 3, 3])), deg=_log(rng, 40, 300),
                    lo=lo, hi=lo + rng.uniform(0.002, 0.05))
    if kind == "random":
        lo = rng.uniform(0.1, 0.8)
        return dict(kind="filter", matrix="random", n=_log(rng, 20000, 1000000), half=rng.randint(5, 9),
                    band=_log(rng, 500, 10000), deg=_log(rng, 30, 60), lo=lo, hi=lo + rng.uniform(0.01, 0.05))
    if kind == "dos":
        return dict(kind="dos", grid=_sides(rng, _log(rng, 4000, 900000), rng.choice([2, 3, 3])),
                    mdeg=_log(rng, 60, 300), nvec=rng.randint(4, 30))
    if kind == "landos":
        return dict(kind="landos", grid=_sides(rng, _log(rng, 4000, 200000)), msteps=rng.randint(20, 40),
                    nvec=rng.randint(4, 20), npts=rng.randint(100, 300))
    if kind == "bounds":
        return dict(kind="bounds", grid=_sides(rng, _log(rng, 4000, 900000), rng.choice([2, 3, 3])),
                    lanm=rng.randint(30, 50), maxit=rng.randint(100, 200))
    if kind in ("run", "mixed"):
        mixed = kind == "mixed"
        s = rng.randint(2, 3) if mixed else rng.randint(2, 5)
        return dict(kind="run", grid=_sides(rng, _log(rng, 3000, 4500 if mixed else 9000)),
                    first=rng.randint(40, 80), count=20 * s, slices=s, nvec=rng.randint(10, 30 if mixed else 60),
                    mdeg=_log(rng, 150, 300), mixed=mixed)
    if kind == "slice":
        return dict(kind="slice", grid=_sides(rng, _log(rng, 8000, 250000)), first=rng.randint(60, 150),
                    count=rng.randint(8, 20))
    if kind == "multi":
        return dict(kind="multi", grids=",".join([_sides(rng, _log(rng, 70000, 200000)),
                                                  _sides(rng, _log(rng, 8000, 30000), 2),
                                                  _sides(rng, _log(rng, 8000, 25000))]),
                    first=rng.randint(40, 80), count=rng.randint(8, 14), slices=rng.randint(2, 3))
    if kind == "gen":
        return dict(kind="gen", grid=_sides(rng, _log(rng, 2000, 7500)), first=rng.randint(20, 30),
                    count=rng.randint(6, 8), slices=2)
    return dict(kind="learned", moments=rng.choice([200, 250, 300]), width=rng.choice([128, 256]),
                layers=rng.randint(3, 4), batch=_log(rng, 33, 1024), steps=rng.randint(2, 8))


# ---------------------------------------------------------------- inputs
def _grid(text):
    return tuple(int(t) for t in text.split("x"))


def _axis(n):
    """Eigenvalues of the 1D Dirichlet Laplacian of n points."""
    return 4.0 * np.sin(np.arange(1, n + 1) * (0.5 * np.pi / (n + 1))) ** 2


def _spectrum(grid):
    """All eigenvalues of laplacian(*grid), in the grid's order (z, y, x)."""
    nx, ny, nz = grid
    x, y = _axis(nx), _axis(ny)
    z = _axis(nz) if nz > 1 else np.zeros(1)
    return (z[:, None, None] + y[None, :, None] + x[None, None, :]).ravel()


def _top(grid):
    """The Gershgorin end of the spectrum."""
    return 12.0 if grid[2] > 1 else 8.0


def _edges(ev, first, count, slices):
    """Ends of `slices` slices of `count` eigenvalues each (ev ascending), from
    near ev[first] on: midpoints of gaps, from the window whose closest
    eigenvalues lie furthest apart."""
    m = count * slices
    top = min(len(ev) - 2, first + 4 * m)
    part = ev[first - 2:top + 2]
    gaps = np.diff(part)
    starts = range(1, max(2, len(gaps) - m - 1))
    i0 = max(starts, key=lambda s: gaps[s - 1:s + m + 1].min())
    i0 = min(i0, len(gaps) - m - 1)
    at = [i0 + count * k for k in range(slices + 1)]
    return [0.5 * (part[i] + part[i + 1]) for i in at], part[i0 + 1:i0 + m + 1]


def _random_matrix(case, seed):
    """Symmetric, `half` draws per row at offsets within the band, values
    N(0,1), diagonal 4 + U[0,1]; CSR on the host and the Gershgorin bounds."""
    n, h, band = case["n"], case["half"], case["band"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    i = torch.arange(n, device=DEV).repeat_interleave(h)
    off = torch.randint(1, band + 1, (n * h,), generator=g, device=DEV)
    j = i + torch.where(torch.rand(n * h, generator=g, device=DEV) < 0.5, -off, off)
    keep = (j >= 0) & (j < n)
    key = torch.unique((torch.minimum(i, j) * n + torch.maximum(i, j))[keep])
    v = torch.randn(key.numel(), generator=g, device=DEV, dtype=torch.float64)
    d = 4.0 + torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    lo, hi, own = key // n, key % n, torch.arange(n, device=DEV)
    rows, cols, vals = torch.cat([lo, hi, own]), torch.cat([hi, lo, own]), torch.cat([v, v, d])
    order = torch.argsort(rows * n + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]
    ia = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ia[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    rad = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, torch.cat([lo, hi]), torch.cat([v, v]).abs())
    return (n, ia.to(torch.int32).cpu().numpy(), cols.to(torch.int32).cpu().numpy(), vals.cpu().numpy(),
            float((d - rad).min()), float((d + rad).max()))


def _step_filter(deg, lmin, lmax, lo, hi):
    """Jackson-damped Chebyshev coefficients of the indicator of the interval
    at fractions lo, hi of [lmin, lmax]: (mu, centre, half width)."""
    cc, dd = 0.5 * (lmin + lmax), 0.5 * (lmax - lmin)
    ta, tb = math.acos(2.0 * lo - 1.0), math.acos(2.0 * hi - 1.0)
    k = np.arange(1, deg + 1)
    q = np.pi / (deg + 2)
    jac = np.sin((k + 1) * q) / ((deg + 2) * math.sin(q)) + (1.0 - (k + 1) / (deg + 2)) * np.cos(k * q)
    mu = np.concatenate([[(ta - tb) / np.pi], 2.0 / np.pi * (np.sin(k * ta) - np.sin(k * tb)) / k * jac])
    return mu, cc, dd


def _start(n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(n, generator=g, device=DEV, dtype=torch.float64)


def _mlp_data(case, seed):
    """Standardised moment pairs and weights U(-1/sqrt K, 1/sqrt K)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    m, w, L, B, S = (case[k] for k in ("moments", "width", "layers", "batch", "steps"))
    X = torch.randn(S + 1, B, m, generator=g, device=DEV)
    T = 0.3 * X + 0.5 * torch.randn(S + 1, B, m, generator=g, device=DEV)
    dims = [m] + [w] * (L - 1) + [m]
    W = [(2.0 * torch.rand(dims[l + 1], dims[l], generator=g, device=DEV) - 1.0) / math.sqrt(dims[l])
         for l in range(L)]
    return X, T, W


def _mlp_layout(W, b):
    """The parameter block: per layer the weights and then the bias, both
    sides padded with zeros to multiples of 16."""
    out = []
    for w, bias in zip(W, b):
        N, K = (-(-s // 16) * 16 for s in w.shape)
        full = torch.zeros(N, K, dtype=w.dtype, device=w.device)
        full[:w.shape[0], :w.shape[1]] = w
        fb = torch.zeros(N, dtype=w.dtype, device=w.device)
        fb[:w.shape[0]] = bias
        out += [full.ravel(), fb]
    return torch.cat(out)


class State:
    """One prepared case: library handles and the call."""

    def __init__(self, case, seed):
        self.case, self.seed, self.lib = case, seed, pv.load()
        self.mats, self.evs, self.held = [], [], []
        getattr(self, "prepare_" + case["kind"])()

    def matrix(self, n, ia, ja, a):
        self.mats.append(pv.Matrix.from_csr(n, ia, ja, a))
        return self.mats[-1]

    def instance(self, A):
        self.evs.append(pv.Instance(A))
        return self.evs[-1]

    def vector(self, n, seed):
        v = pv.Vector(n, _start(n, seed).cpu().numpy())
        self.held.append(v)
        return v

    def __del__(self):
        for ev in self.evs:
            ev.close()
        for x in self.held:
            x.close() if isinstance(x, pv.Mlp) else x.free()
        for m in self.mats:
            m.free()

    # one filter application, vectors on the device
    def prepare_filter(self):
        c = self.case
        if c["matrix"] == "grid":
            n, ia, ja, a = laplacian(*_grid(c["grid"]))
            lmin, lmax = 0.0, _top(_grid(c["grid"]))
        else:
            n, ia, ja, a, lmin, lmax = _random_matrix(c, self.seed)
        self.ev = self.instance(self.matrix(n, ia, ja, a))
        mu, cc, dd = _step_filter(c["deg"], lmin, lmax, c["lo"], c["hi"])
        self.pol, self.keep = pv._polparams(pv.Filter(1, c["deg"], 0.0, 0.5, cc, dd, mu))
        self.x = _start(n, self.seed + 1)
        self.y = torch.empty_like(self.x)

    def run_filter(self):
        st = self.lib.pEVSL_B200_ChebAv(self.ev.p, C.byref(self.pol), self.x.data_ptr(), self.y.data_ptr())
        if st:
            raise RuntimeError("pEVSL_B200_ChebAv returned %d" % st)
        return self.y

    # KPM density of states
    def prepare_dos(self):
        g = _grid(self.case["grid"])
        self.ev = self.instance(self.matrix(*laplacian(*g)))
        self.intv = [0.1, 0.25 * _top(g), 0.0, _top(g)]

    def run_dos(self):
        pv.set_rng(pv.RNG_GAUSS, self.seed)
        st, mu, count = self.ev.kpmdos(self.case["mdeg"], 1, self.case["nvec"], self.intv)
        if st:
            raise RuntimeError("pEVSL_Kpmdos returned %d" % st)
        return {"mu": mu, "count": np.float64(count)}

    # Lanczos density of states
    prepare_landos = prepare_dos

    def run_landos(self):
        c = self.case
        pv.set_rng(pv.RNG_GAUSS, self.seed)
        st, xd, yd, count = self.ev.landos(c["nvec"], c["msteps"], c["npts"], self.intv)
        if st:
            raise RuntimeError("pEVSL_LanDosG returned %d" % st)
        return {"x": xd, "dos": yd, "count": np.float64(count)}

    # spectrum bounds
    def prepare_bounds(self):
        A = self.matrix(*laplacian(*_grid(self.case["grid"])))
        self.ev, self.v = self.instance(A), self.vector(A.n, self.seed)

    def run_bounds(self):
        lo, hi = C.c_double(), C.c_double()
        st = self.lib.pEVSL_LanTrbounds(self.ev.p, self.case["lanm"], self.case["maxit"], 1e-8, C.byref(self.v.pv),
                                        1, C.byref(lo), C.byref(hi), None)
        if st:
            raise RuntimeError("pEVSL_LanTrbounds returned %d" % st)
        return np.array([lo.value, hi.value])

    # a whole run over an interval
    def prepare_run(self):
        c, g = self.case, _grid(self.case["grid"])
        ends, _ = _edges(np.sort(_spectrum(g)), c["first"], c["count"], 1)
        self.A = self.matrix(*laplacian(*g))
        self.s = pv.SliceRun(ends[0], ends[-1], c["slices"], lmin=0.0, lmax=_top(g), Mdeg=c["mdeg"], nvec=c["nvec"],
                             rng_mode=pv.RNG_GAUSS, seed=self.seed)

    def run_run(self):
        r = pv.solve_interval(self.A, self.s, batched=True,
                              precision=pv.PREC_MIXED if self.case["mixed"] else pv.PREC_FP64)
        if r.status:
            raise RuntimeError("solve_interval returned %d" % r.status)
        return np.sort(np.concatenate(r.lam))

    # slices of one or several problems
    def problem(self, g, first, count, slices, mass=False):
        ev_all = np.sort(_pencil(_spectrum(g), mass))
        ends, _ = _edges(ev_all, first, count, slices)
        n, ia, ja, a = laplacian(*g)
        A = self.matrix(n, ia, ja, a)
        ev = self.instance(A)
        lmin, lmax = 0.0, float(_pencil(np.array([_top(g)]), mass)[0])
        ivs = [[ends[k], ends[k + 1], lmin, lmax] for k in range(slices)]
        filters = []
        for iv in ivs:
            code, f = pv.findpol(iv)
            if code:
                raise RuntimeError("pEVSL_FindPol returned %d" % code)
            filters.append(f)
        mlan = min(max(5 * (count + 2), 300), n)
        v = self.vector(n, self.seed + len(self.evs))
        return A, (ev, ivs, [mlan] * slices, 1e-8, v, filters), (n, ia, ja, a)

    def prepare_slice(self):
        c = self.case
        _, self.p, _ = self.problem(_grid(c["grid"]), c["first"], c["count"], 1)

    def run_slice(self):
        ev, ivs, mx, tol, v, filters = self.p
        out = ev.cheblannr(ivs[0], mx[0], tol, v, filters[0])
        if out["status"]:
            raise RuntimeError("pEVSL_ChebLanNr returned %d" % out["status"])
        return out["lam"]

    def prepare_multi(self):
        c = self.case
        self.ps = [self.problem(_grid(g), c["first"], c["count"], c["slices"])[1] for g in c["grids"].split(",")]

    def run_multi(self):
        st, outs = pv.cheblannr_multi(self.ps)
        if st:
            raise RuntimeError("pEVSL_B200_ChebLanNrMulti returned %d" % st)
        return [[s["lam"] for s in p] for p in outs]

    # a generalized problem; B = (12 I + neighbours) / 18
    def prepare_gen(self):
        c = self.case
        _, self.p, (n, ia, ja, a) = self.problem(_grid(c["grid"]), c["first"], c["count"], c["slices"], mass=True)
        B = self.matrix(n, ia, ja, np.where(a > 0, 12.0 / 18.0, 1.0 / 18.0))
        bsol = pv.BSolver(B, "lsrec", 1.0 / 3.0, 1.0, 80, 1e-10)
        self.held.append(bsol)
        self.p[0].set_generalized(B, bsol)

    def run_gen(self):
        ev, ivs, mx, tol, v, filters = self.p
        st, outs = pv.cheblannr_batch(ev, ivs, mx, tol, v, filters)
        if st:
            raise RuntimeError("pEVSL_B200_ChebLanNrBatch returned %d" % st)
        return [s["lam"] for s in outs]

    # training steps and a prediction of the learned density of states
    def prepare_learned(self):
        c = self.case
        self.X, self.T, W = _mlp_data(c, self.seed)
        self.net = pv.Mlp(c["moments"], c["width"], c["moments"], c["layers"])
        self.held.append(self.net)
        p = _mlp_layout(W, [torch.zeros(w.shape[0], device=DEV) for w in W])
        self.net.set_params(p.cpu().numpy())
        self.Y = torch.empty(c["batch"], c["moments"], device=DEV)

    def run_learned(self):
        c, loss, losses = self.case, C.c_float(), []
        for s in range(c["steps"]):
            st = self.lib.pEVSL_B200_MlpTrainStep(self.net.p, self.X[s].data_ptr(), self.T[s].data_ptr(), c["batch"],
                                                  1e-3, C.byref(loss))
            if st:
                raise RuntimeError("pEVSL_B200_MlpTrainStep returned %d" % st)
            losses.append(loss.value)
        st = self.lib.pEVSL_B200_MlpForward(self.net.p, self.X[-1].data_ptr(), self.Y.data_ptr(), c["batch"])
        if st:
            raise RuntimeError("pEVSL_B200_MlpForward returned %d" % st)
        return {"loss": np.array(losses, np.float32), "params": self.net.get_params(), "pred": self.Y}


def prepare(case, seed):
    return State(case, seed)


def run(state):
    return getattr(state, "run_" + state.case["kind"])()


# ---------------------------------------------------------------- work
def _entries(g):
    nx, ny, nz = g
    n = nx * ny * nz
    faces = 2 * ((nx - 1) * ny * nz + nx * (ny - 1) * nz + (nx * ny * (nz - 1) if nz > 1 else 0))
    return n, n + faces


def work(case):
    """The matrix, the start vectors and the results once; the operations of
    the recurrences where their number is given by the case.  A solve's step
    count is found by the run: it is taken as four per eigenvalue, with the
    projections on the basis, and its filter as at least one product."""
    k = case["kind"]
    if k == "learned":
        m, w, L, B, S = (case[x] for x in ("moments", "width", "layers", "batch", "steps"))
        np_ = 2 * m * w + (L - 2) * w * w + (L - 1) * w + m
        return {"bytes": 4.0 * (2 * np_ * 3 + 2 * (S + 1) * B * m), "flops": 2.0 * np_ * B * (3 * S + 1)}
    if k == "filter" and case["matrix"] == "random":
        n, nnz = case["n"], case["n"] * (2 * case["half"] + 1)
    else:
        n, nnz = _entries(_grid(case["grid"])) if k != "multi" else (0, 0)
    mat = 12.0 * nnz + 4.0 * (n + 1)
    if k == "filter":
        return {"bytes": mat + 16.0 * n, "flops": case["deg"] * (2.0 * nnz + 6.0 * n)}
    if k == "dos":
        return {"bytes": mat + 8.0 * n * case["nvec"], "flops": case["mdeg"] * case["nvec"] * (2.0 * nnz + 6.0 * n)}
    if k == "landos":
        s = case["msteps"]
        return {"bytes": mat + 8.0 * n * case["nvec"], "flops": case["nvec"] * s * (2.0 * nnz + 2.0 * n * s)}
    if k == "bounds":
        return {"bytes": mat + 8.0 * n, "flops": case["maxit"] * (2.0 * nnz + 2.0 * n * case["lanm"])}
    if k == "run":
        st = 4 * case["count"]
        return {"bytes": mat + 8.0 * n * (case["nvec"] + 1 + case["count"]),
                "flops": st * 2.0 * nnz + case["mdeg"] * case["nvec"] * (2.0 * nnz + 6.0 * n)}
    total = {"bytes": 0.0, "flops": 0.0}
    for g in (case["grids"].split(",") if k == "multi" else [case["grid"]]):
        n, nnz = _entries(_grid(g))
        per, slices = case["count"], case.get("slices", 1)
        total["bytes"] += 12.0 * nnz + 4.0 * (n + 1) + 8.0 * n * (1 + per * slices)
        total["flops"] += slices * 4 * per * (2.0 * nnz + 4.0 * n * 2 * per)
    return total


# ---------------------------------------------------------------- results in 64 bits
def _pencil(lam, mass):
    """Eigenvalues of the pencil (A, (12 I + neighbours) / 18), 3D grids: the
    neighbours' sum is 6 I - A, so B has the eigenvalues (18 - lam) / 18."""
    return lam / ((18.0 - lam) / 18.0) if mass else lam


def _sines(n):
    """The orthonormal eigenvectors of the 1D Dirichlet Laplacian."""
    i = torch.arange(1, n + 1, device=DEV)
    q = (i[:, None] * i[None, :]) % (2 * (n + 1))
    return torch.sin(q.double() * (math.pi / (n + 1))) * math.sqrt(2.0 / (n + 1))


def _to_modes(v, g):
    """Coefficients of v (its own inverse) on the grid's eigenvectors."""
    nx, ny, nz = g
    t = v.reshape(nz, ny, nx)
    t = torch.einsum("zyx,xa->zya", t, _sines(nx))
    t = torch.einsum("zya,yb->zba", t, _sines(ny))
    if nz > 1:
        t = torch.einsum("zba,zc->cba", t, _sines(nz))
    return t.reshape(-1)


def _philox_gauss(n, nvec, seed):
    """The library's Gaussian stream, draws 0 .. nvec-1 of length n: Philox
    4x32-10 (Salmon et al., 2011) and Box-Muller on 53-bit uniforms."""
    mask = 0xffffffff
    p = torch.arange((n + 1) // 2, device=DEV, dtype=torch.int64)
    for m in range(nvec):
        c = [p & mask, p >> 32, torch.full_like(p, m), torch.zeros_like(p)]
        k0, k1 = seed & mask, (seed >> 32) & mask
        for _ in range(10):
            a, b = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
            c = [((b >> 32) & mask) ^ c[1] ^ k0, b & mask, ((a >> 32) & mask) ^ c[3] ^ k1, a & mask]
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        u = [(((hi << 21) | (lo >> 11)) & ((1 << 53) - 1)).double() for hi, lo in ((c[0], c[1]), (c[2], c[3]))]
        rad = torch.sqrt(-2.0 * torch.log((u[0] + 0.5) / 2.0 ** 53))
        ang = (2.0 * math.pi) * (u[1] / 2.0 ** 53)
        yield torch.stack([rad * torch.cos(ang), rad * torch.sin(ang)], 1).reshape(-1)[:n]


def _csr(n, ia, ja, a):
    return torch.sparse_csr_tensor(torch.from_numpy(ia), torch.from_numpy(ja), torch.from_numpy(a), (n, n),
                                   dtype=torch.float64, device=DEV)


def _exact_filter(case, seed):
    if case["matrix"] == "grid":
        g = _grid(case["grid"])
        mu, cc, dd = _step_filter(case["deg"], 0.0, _top(g), case["lo"], case["hi"])
        x = (torch.from_numpy(_spectrum(g)).to(DEV) - cc) / dd
        b1, b2 = torch.zeros_like(x), torch.zeros_like(x)
        for k in range(case["deg"], 0, -1):
            b1, b2 = mu[k] + 2.0 * x * b1 - b2, b1
        p = mu[0] + x * b1 - b2
        v = _start(x.numel(), seed + 1)
        return _to_modes(p * _to_modes(v, g), g)
    n, ia, ja, a, lmin, lmax = _random_matrix(case, seed)
    mu, cc, dd = _step_filter(case["deg"], lmin, lmax, case["lo"], case["hi"])
    A, v = _csr(n, ia, ja, a), _start(n, seed + 1)
    vk, vm, y = (A @ v - cc * v) / dd, v, mu[0] * v
    y = y + mu[1] * vk
    for k in range(2, case["deg"] + 1):
        vk, vm = 2.0 / dd * (A @ vk - cc * vk) - vm, vk
        y = y + mu[k] * vk
    return y


def _exact_dos(case, seed):
    g = _grid(case["grid"])
    lam, top, M = torch.from_numpy(_spectrum(g)).to(DEV), _top(g), case["mdeg"]
    w = torch.zeros_like(lam)
    for v in _philox_gauss(lam.numel(), case["nvec"], seed):
        w += _to_modes(v / torch.linalg.norm(v), g) ** 2
    theta = torch.arccos(lam / (0.5 * top) - 1.0)
    k = np.arange(1, M + 1)
    q = np.pi / (M + 2)
    jac = np.sin((k + 1) * q) / ((M + 2) * math.sin(q)) + (1.0 - (k + 1) / (M + 2)) * np.cos(k * q)
    dots = np.array([float((w * torch.cos(i * theta)).sum()) for i in k])
    mu = np.concatenate([[float(case["nvec"])], 2.0 * jac * dots]) / (case["nvec"] * math.pi)
    b = [math.acos(t / (0.5 * top) - 1.0) for t in (0.1, 0.25 * top)]
    tcnt = -mu[0] * (b[1] - b[0]) - float(np.sum(mu[1:] * (np.sin(k * b[1]) - np.sin(k * b[0])) / k))
    return {"mu": mu, "count": np.float64(tcnt * lam.numel())}


def _exact_landos(case, seed):
    g, m, npts = _grid(case["grid"]), case["msteps"], case["npts"]
    n, ia, ja, a = laplacian(*g)
    A, top = _csr(n, ia, ja, a), _top(g)
    x = np.linspace(0.1, 0.25 * top, npts)
    y = np.zeros(npts)
    sigma = top / (min(m, 30) - 1) / math.sqrt(8.0 * math.log(1.25))
    width = sigma * math.sqrt(-2.0 * math.log(1e-8))
    for v in _philox_gauss(n, case["nvec"], seed):
        V = torch.zeros(m + 1, n, dtype=torch.float64, device=DEV)
        V[0] = v / torch.linalg.norm(v)
        T = np.zeros((m, m))
        for k in range(m):
            w = A @ V[k]
            T[k, k] = float(torch.dot(w, V[k]))
            for _ in range(2):
                w = w - V[:k + 1].T @ (V[:k + 1] @ w)
            b = float(torch.linalg.norm(w))
            V[k + 1] = w / b
            if k + 1 < m:
                T[k, k + 1] = T[k + 1, k] = b
        th, S = np.linalg.eigh(T)
        d = x[None, :] - th[:, None]
        y += np.sum(np.where(np.abs(d) < width, S[0][:, None] ** 2 * np.exp(-d * d / (2.0 * sigma ** 2)), 0.0), 0)
    y /= case["nvec"] * math.sqrt(2.0 * sigma ** 2 * math.pi)
    return {"x": x, "dos": y, "count": None}


def _exact_learned(case, seed):
    X, T, W = _mlp_data(case, seed)
    P = [t for w in W for t in (w.double().requires_grad_(), torch.zeros(w.shape[0], dtype=torch.float64, device=DEV,
                                                                         requires_grad=True))]
    opt = torch.optim.Adam(P, lr=1e-3, betas=(0.9, 0.999), eps=1e-8)

    def net(x):
        for l in range(len(W)):
            x = x @ P[2 * l].T + P[2 * l + 1]
            x = torch.nn.functional.gelu(x) if l + 1 < len(W) else x
        return x

    losses = []
    for s in range(case["steps"]):
        opt.zero_grad()
        loss = ((net(X[s].double()) - T[s].double()) ** 2).mean()
        loss.backward()
        opt.step()
        losses.append(float(loss))
    with torch.no_grad():
        return {"loss": np.array(losses), "params": _mlp_layout(P[0::2], P[1::2]).detach().cpu().numpy(),
                "pred": net(X[-1].double())}


def exact(case, seed):
    k = case["kind"]
    if k in ("filter", "dos", "landos", "learned"):
        return globals()["_exact_" + k](case, seed)
    if k == "bounds":
        # enclosures with a residual's margin, not eigenvalues: nothing to be near to
        return None
    if k == "run":
        return _edges(np.sort(_spectrum(_grid(case["grid"]))), case["first"], case["count"], 1)[1]
    out = []
    for g in (case["grids"].split(",") if k == "multi" else [case["grid"]]):
        count, slices = case["count"], case.get("slices", 1)
        lam = _edges(np.sort(_pencil(_spectrum(_grid(g)), k == "gen")), case["first"], count, slices)[1]
        out.append([lam[i * count:(i + 1) * count] for i in range(slices)])
    return out if k == "multi" else out[0] if k == "gen" else out[0][0]
