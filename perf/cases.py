"""The work that users of the tracking library have it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a user's program has
in hand before the call (models, releases, handles), ``run`` is one pass
through the public entry points of ``mprw`` and returns everything it
computes, ``work`` the bytes and operations one pass cannot do without, and
``exact`` the values of ``run`` in 64 bits from plain torch, where the outputs
are a formula of the inputs (reconstructions, gradients).  The trajectories of
the random walk have no such formula (every step depends on all before it).
"""
from __future__ import annotations

import math
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "modpath-rw_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mprw  # noqa: E402
from mprw import workloads as W  # noqa: E402
from mprw.model import (ACTIVE, EULERIAN, EXPONENTIAL, FP64, MIN_ADV_DISP, MIXED, Options, Particles)  # noqa: E402


def listed():
    return [
        # A plume in a uniform column (the analytic test problem), few particles, its 1-D concentration at
        # every time point: the smallest calls, where launches and host reads count.
        dict(name="column_small", kind="column", n=1000, intervals=4, days=5.0, precision="fp64"),
        # The headline workload: a million particles in the lognormal slab, tracked over three intervals.
        dict(name="slab_fp64", kind="walk", ncol=200, nrow=100, nlay=20, n=1_000_000, intervals=3, days=10.0,
             precision="fp64", exponential=False, axisymmetric=False),
        # The same slab in mixed precision (the production setting for ensembles), over five intervals.
        dict(name="slab_mixed", kind="walk", ncol=200, nrow=100, nlay=20, n=1_000_000, intervals=5, days=10.0,
             precision="mixed", exponential=False, axisymmetric=False),
        # An odd-sized aquifer with the other transport options: exponential in-cell advection with its Newton
        # exit time, axisymmetric dispersion.
        dict(name="aquifer_exp_axi", kind="walk", ncol=61, nrow=37, nlay=7, n=40_001, intervals=2, days=5.0,
             precision="fp64", exponential=True, axisymmetric=True),
        # A transient flow model: each time step loads new flows, moves a modest release one day and records its
        # sink and resident observations.
        dict(name="transient_step", kind="flow", ncol=200, nrow=100, nlay=20, n=50_000, days=1.0),
        # Reconstruction of a plume's concentration on the 1 m grid, double precision (the reference's).
        dict(name="kde3d_fp64", kind="kde", ncol=200, nrow=100, nlay=20, n=1_000_000, days=80.0, precision="fp64",
             weighted=False),
        # The same in single precision, fewer particles, ragged grid.
        dict(name="kde3d_mixed", kind="kde", ncol=187, nrow=93, nlay=21, n=300_000, days=60.0, precision="mixed",
             weighted=False),
        # A plan-view (2-D) reconstruction of particles that carry solute masses.
        dict(name="kde2d_weighted", kind="kde", ncol=250, nrow=50, nlay=1, n=250_000, days=80.0, precision="fp64",
             weighted=True),
        # A small ensemble in one batch, mixed precision: advance all, reconstruct every member.
        dict(name="ensemble_mixed", kind="batch", members=6, n=400_000, intervals=2, days=10.0),
        # A few realizations of the ensemble generator's smallest grids in double precision.
        dict(name="ensemble_fp64_small", kind="batch", members=3, n=30_000, intervals=1, days=10.0, precision="fp64"),
        # Gradient of a concentration misfit for calibration: the differentiable walk forward and its adjoint.
        dict(name="adjoint_slab", kind="adjoint", ncol=100, nrow=50, nlay=10, n=100_000, nsteps=200, checkpoint=20),
        # Breakthrough curve of a well: the 1-D reconstruction of a million arrival records.
        dict(name="btc_1e6", kind="series", n=1_000_000, bin_format=1, fraction=0.75, eff_format=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["column", "walk", "walk", "flow", "kde", "kde", "batch", "adjoint", "series"])
    grid = dict(ncol=rng.randint(40, 200), nrow=rng.randint(20, 100), nlay=rng.randint(5, 20))
    prec = rng.choice(["fp64", "mixed"])
    if kind == "column":
        return dict(kind=kind, n=_log_int(rng, 500, 100_000), intervals=rng.randint(2, 4),
                    days=round(rng.uniform(2.0, 8.0), 1), precision=prec)
    if kind == "walk":
        exp, axi = rng.random() < 0.25, rng.random() < 0.25
        return dict(kind=kind, **grid, n=_log_int(rng, 5_000, 40_000 if exp else 1_000_000),
                    intervals=rng.randint(1, 2 if exp else 3), precision=prec, exponential=exp, axisymmetric=axi,
                    days=round(rng.uniform(2.0, 5.0) if exp else rng.uniform(5.0, 10.0), 1))
    if kind == "flow":
        return dict(kind=kind, **grid, n=_log_int(rng, 2_000, 50_000), days=round(rng.uniform(0.5, 1.5), 2))
    if kind == "kde":
        flat = rng.random() < 0.3
        if flat:
            grid.update(nlay=1, ncol=rng.randint(80, 250))
        return dict(kind=kind, **grid, n=_log_int(rng, 20_000, 1_000_000 if not flat else 250_000),
                    days=round(rng.uniform(20.0, 80.0), 1), precision=prec, weighted=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(2, 6), n=_log_int(rng, 10_000, 400_000), intervals=1,
                    days=round(rng.uniform(5.0, 10.0), 1), precision=prec)
    if kind == "adjoint":
        return dict(kind=kind, ncol=rng.randint(30, 100), nrow=rng.randint(20, 50), nlay=rng.randint(4, 10),
                    n=_log_int(rng, 2_000, 100_000), nsteps=rng.randint(40, 200), checkpoint=rng.randint(7, 25))
    return dict(kind=kind, n=_log_int(rng, 20_000, 1_000_000), bin_format=rng.choice([0, 1]),
                fraction=round(rng.uniform(0.5, 1.2), 2), eff_format=rng.choice([0, 2, 3]))


# ---- inputs --------------------------------------------------------------------
@lru_cache(maxsize=16)
def _model(ncol, nrow, nlay, field=0, sigma2=1.0, alpha_l=0.5):
    """Grid and steady flow of the lognormal generator (a model is built once per program)."""
    g, f, _ = W.heterogeneous_flow(nlay, nrow, ncol, sigma2=sigma2, kg=10.0, lh=10.0, lv=2.0, porosity=0.25,
                                   alpha_l=alpha_l, alpha_t=alpha_l / 10.0, dm=1e-4, seed=field)
    return g, f


def _precision(case):
    return MIXED if case.get("precision", "mixed") == "mixed" else FP64


def _release(g, n, seed, x1=10.0, status=0):
    return W.release_in_box(g, n, 0.0, min(x1, float(g.ncol)), 0.0, float(g.nrow), float(g.botm[-1]),
                            float(g.top[0]), seed=seed, status=status)


def _plume(case, seed):
    """A plume of stream tubes: inlet-slab releases carried by a smooth lognormal velocity per (y, z) with
    longitudinal dispersion -- the fingered shape that tracking a lognormal field gives.  Returns the
    particles and their model coordinates."""
    rng = np.random.default_rng(seed)
    n, ncol, nrow, nlay, t = case["n"], case["ncol"], case["nrow"], case["nlay"], case["days"]
    ny, nz = 2 * nrow, 2 * nlay
    ky = np.fft.fftfreq(ny)[None, :] * 2.0 * math.pi * 6.0
    kz = np.fft.fftfreq(nz)[:, None] * 2.0 * math.pi * 1.2
    z = np.fft.ifft2(np.fft.fft2(rng.standard_normal((nz, ny))) * np.exp(-0.25 * (ky ** 2 + kz ** 2))).real
    v = 0.2 * np.exp(0.5 * z / z.std())
    Y, Z = rng.uniform(0.0, nrow, n), rng.uniform(0.0, nlay, n)
    vt = v[np.minimum(Z.astype(int), nlay - 1), np.minimum(Y.astype(int), nrow - 1)] * t
    X = rng.uniform(0.0, 10.0, n) + vt + np.sqrt(vt) * rng.standard_normal(n)
    X = np.abs(X)
    X = np.minimum(np.where(X > ncol, 2.0 * ncol - X, X), ncol - 1e-6)
    X, Y, Z = np.maximum(X, 0.0), np.minimum(Y, nrow - 1e-9), np.minimum(Z, nlay - 1e-9)
    j, i, k = X.astype(np.int64), nrow - 1 - Y.astype(np.int64), nlay - 1 - Z.astype(np.int64)
    lx, ly, lz = X - np.floor(X), Y - np.floor(Y), Z - np.floor(Z)
    # the model coordinates of the stored local ones, as the grid maps them
    xyz = np.stack([(1.0 - lx) * j + lx * (j + 1.0), (1.0 - ly) * (nrow - 1.0 - i) + ly * (nrow - i * 1.0),
                    (1.0 - lz) * (nlay - 1.0 - k) + lz * (nlay - k * 1.0)], 1)
    mass = rng.lognormal(0.0, 0.5, n) if case["weighted"] else np.ones(n)
    p = Particles(cell=(k * nrow * ncol + i * ncol + j + 1).astype(np.int32), lx=lx, ly=ly, lz=lz, t=np.full(n, t),
                  status=np.full(n, ACTIVE, np.int32), mass=mass, id=np.arange(n, dtype=np.uint64),
                  rng_ctr=np.zeros(n, np.uint64))
    return p, xyz


def _options(case, seed):
    return Options(time_step_kind=MIN_ADV_DISP, ts_param=(0.1, 0.1),
                   advection_kind=EXPONENTIAL if case.get("exponential") else EULERIAN,
                   dispersion_model=1 if case.get("axisymmetric") else 0, stop_weak_sinks=True,
                   rng_seed=0x5EED + seed, precision=_precision(case))


def _arrivals(case, seed):
    """Arrival times and masses of a breakthrough: lognormal travel times of two pathways."""
    rng = np.random.default_rng(seed)
    n, m = case["n"], int(0.3 * case["n"])
    # stratified: the quartiles, and with them the automatic bin size, are the same distribution's at every seed
    u = np.concatenate([(np.arange(m) + rng.uniform(0.0, 1.0, m)) / m,
                        (np.arange(n - m) + rng.uniform(0.0, 1.0, n - m)) / (n - m)])
    z = math.sqrt(2.0) * torch.erfinv(2.0 * torch.as_tensor(u) - 1.0).clamp(-4.0, 4.0).numpy()
    slow = np.arange(n) < m
    t = np.exp(np.where(slow, math.log(180.0) + 0.25 * z, math.log(90.0) + 0.35 * z))
    t = t[rng.permutation(n)]
    return t, rng.uniform(0.5, 1.5, n)


def _batch_members(case):
    """Member k: an odd-sized grid of the lognormal generator with its own variance and dispersivity; the
    particle counts shrink geometrically from n."""
    return [dict(ncol=101 + 23 * k, nrow=60 - 7 * k, nlay=10 + k, sigma2=0.5 + 0.25 * k, alpha_l=0.1 + 0.15 * k,
                 n=max(1000, int(case["n"] * 0.7 ** k))) for k in range(case["members"])]


def _zones(g):
    k, i, j = np.unravel_index(np.arange(g.ncell), (g.nlay, g.nrow, g.ncol))
    return ((j >= g.ncol // 2).astype(np.int32) + 2 * (i >= g.nrow // 2) + 4 * (k >= g.nlay // 2)).astype(np.int32)


_ADJ = dict(dt=0.05, eps=0.01, h=(2.0, 2.0, 1.0), nz=8)


def _adjoint_inputs(case, seed):
    g, f = _model(case["ncol"], case["nrow"], case["nlay"])
    p = _release(g, case["n"], 4000 + seed, x1=15.0, status=ACTIVE)
    rng = np.random.default_rng(seed)
    fac = rng.uniform(0.95, 1.05, 24)
    theta = np.concatenate([0.5 * fac[:8], 0.05 * fac[8:16], 0.25 * fac[16:], [1.0]])
    # the density gradient of a misfit against smooth observations
    grad = rng.standard_normal((g.nlay, g.nrow, g.ncol))
    return g, f, p, theta, grad


def prepare(case, seed):
    kind, st = case["kind"], dict(case)
    if kind == "column":
        g, f, p, opt = W.uniform_pulse(n_particles=case["n"], precision=_precision(case))
        opt.rng_seed = 0x5EED + seed
        p.lx = np.random.default_rng(seed).uniform(0.0, 1.0, p.n)
    elif kind == "walk":
        g, f = _model(case["ncol"], case["nrow"], case["nlay"])
        if case["axisymmetric"]:
            f = W.Flow(**{**f.__dict__, "alpha_lv": np.array([0.2]), "alpha_tv": np.array([0.01])})
        p, opt = _release(g, case["n"], 1000 + seed), _options(case, seed)
    elif kind == "flow":
        g, f = _model(case["ncol"], case["nrow"], case["nlay"])
        rng = np.random.default_rng(seed)
        # the next time step of the flow model: all flows scaled, storage porosity of every cell its own
        s = rng.uniform(0.8, 1.2)
        f = W.Flow(**{**f.__dict__, "flowja": f.flowja * s, "source_flow": f.source_flow * s,
                      "sink_flow": f.sink_flow * s, "porosity": rng.uniform(0.2, 0.3, g.ncell)})
        # released between a resident observation near the inlet and the outlet's constant-head cells
        p = W.release_in_box(g, case["n"], 5.0, float(g.ncol), 0.0, float(g.nrow), float(g.botm[-1]),
                             float(g.top[0]), seed=1000 + seed, status=ACTIVE)
        opt = _options(dict(precision="fp64"), seed)
        col = np.arange(g.ncell) % g.ncol
        cells = np.concatenate([np.where(col == g.ncol // 2)[0], np.where(col == g.ncol - 1)[0]]) + 1
        st["obs"] = (cells, np.repeat([0, 1], [cells.size // 2, cells.size // 2]), np.array([1, 2]))
    elif kind == "kde":
        g = W.structured_grid(case["nlay"], case["nrow"], case["ncol"])
        p, _ = _plume(case, seed)
        f, opt = None, _options(case, seed)
    elif kind == "batch":
        mem = _batch_members(case)
        models = [_model(m["ncol"], m["nrow"], m["nlay"], k, m["sigma2"], m["alpha_l"]) for k, m in enumerate(mem)]
        b = mprw.Batch([g for g, _ in models], _options(case, seed))
        parts = []
        for k, ((g, f), m) in enumerate(zip(models, mem)):
            b.load_flow(k, f)
            p = _release(g, m["n"], 1000 * (k + 1) + seed)
            p.id = (np.uint64(k) << np.uint64(40)) + np.arange(p.n, dtype=np.uint64)
            parts.append(p)
        b.set_particles(parts)
        st.update(b=b, parts=parts, domains=[(float(g.ncol), float(g.nrow), float(g.nlay)) for g, _ in models])
        return st
    elif kind == "adjoint":
        g, f, p, st["theta"], st["grad"] = _adjoint_inputs(case, seed)
        opt = _options(dict(precision="fp64"), seed)
    else:
        st["t"], st["w"] = _arrivals(case, seed)
        return st
    tr = mprw.Tracker(g, opt)
    if f is not None:
        tr.load_flow(f)
    tr.set_particles(p)
    if kind == "flow":
        tr.set_observations(*st["obs"])
    if kind == "adjoint":
        tr.adj_setup(_zones(g), _ADJ["nz"], _ADJ["dt"], case["nsteps"], case["checkpoint"], (0.0, 0.0, 0.0),
                     (1.0, 1.0, 1.0), (g.ncol, g.nrow, g.nlay), _ADJ["h"], _ADJ["eps"], seed=seed)
    st.update(tr=tr, p=p, f=f)
    return st


# ---- one pass ------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "series":
        r = mprw.gpkde_series(st["t"], st["w"], domain_size=400.0, bin_format=st["bin_format"],
                              bin_size_fraction=st["fraction"], init_factor=3.0, eff_format=st["eff_format"])
        return [r["counts"], r["density"], r["bin_size"], r["coordinates"], r["n_bins"], r["loops"],
                r["active_bins"]]
    if kind == "batch":
        b, t = st["b"], 0.0
        b.set_particles(st["parts"])
        steps = 0
        for _ in range(st["intervals"]):
            steps += b.advance(t, t + st["days"])
            t += st["days"]
        dens, loops = b.gpkde(st["domains"], (1.0, 1.0, 1.0), precision=_precision(st))
        return [steps, dens, loops, b.get_particles(global_xyz=False)]
    tr = st["tr"]
    if kind == "adjoint":
        rho = tr.adj_forward(st["theta"])
        return [rho, tr.adj_backward(st["grad"])]
    if kind == "kde":
        dens, hist, loops = tr.gpkde((float(st["ncol"]), float(st["nrow"]), float(st["nlay"])), (1.0, 1.0, 1.0),
                                     precision=_precision(st))
        return [dens, hist, loops]
    out = []
    if kind == "flow":
        tr.load_flow(st["f"])
    tr.set_particles(st["p"])
    steps, t = 0, 0.0
    for _ in range(st.get("intervals", 1)):
        steps += tr.advance(t, t + st["days"])
        t += st["days"]
        if kind == "column":
            dens, hist, loops = tr.gpkde((200.0, 1.0, 1.0), (1.0, 1.0, 1.0), precision=_precision(st))
            out += [dens, hist, loops]
    if kind == "flow":
        rec = tr.observe_sinks()
        arrival = np.zeros(tr.n)  # by particle: when it reached the outlet's observation (0: not yet)
        arrival[rec["id"]] = rec["time"]
        out += [arrival, list(tr.observe_resident())]
    return [steps, tr.get_particles(), out]


# ---- what a pass cannot do without ----------------------------------------------
_STATE = 4 + 4 + 3 * 8 + 8 + 8          # cell, status, local coordinates, time, random counter
_FLOPS_STEP = 145.0                     # floating-point operations of one random-walk step
_PER_DAY = 4.5                          # steps per particle and day of the lognormal generator at Courant 0.1


def _kde_flops(active, ndim, loops=8):
    """Separable smoothing of the active bins alone: per loop, dimension and bin 8 smoothing gathers and 3
    second-derivative scatters of about 13 taps, a density scatter of 7^ndim cells, 200 operations per bin."""
    return loops * active * (2.0 * 13 * 11 * ndim + 2.0 * 7 ** ndim + 200.0)


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "series":
        return dict(bytes=16.0 * n + 24.0 * 560, flops=4.0 * n + 4 * 560 * 60 * 40.0)
    if kind == "kde":
        ncell = case["ncol"] * case["nrow"] * case["nlay"]
        ndim = 3 if case["nlay"] > 1 else 2
        active = min(n, 0.2 * ncell)
        return dict(bytes=(4 + 4 + 24 + 8 * case["weighted"]) * n + 16.0 * ncell,
                    flops=20.0 * n + _kde_flops(active, ndim))
    if kind == "adjoint":
        g = case["ncol"] * case["nrow"] * case["nlay"]
        return dict(bytes=48.0 * n + 16.0 * g, flops=900.0 * n * case["nsteps"])
    if kind == "column":
        m = case["intervals"]
        return dict(bytes=n * (_STATE + 16 + _STATE + 24.0) + m * 16.0 * 200,
                    flops=m * (10.0 * case["days"] * n * _FLOPS_STEP + _kde_flops(60, 1)))
    if kind == "batch":
        mem = _batch_members(case)
        tot = sum(m["n"] for m in mem)
        cells = sum(m["ncol"] * m["nrow"] * m["nlay"] for m in mem)
        return dict(bytes=tot * (2 * _STATE + 16.0) + 8.0 * cells,
                    flops=tot * case["intervals"] * case["days"] * _PER_DAY * _FLOPS_STEP + _kde_flops(0.2 * cells, 3))
    g = case["ncol"] * case["nrow"] * case["nlay"] if kind == "flow" else 0
    # flow: connections, face flows, per-cell arrays in; the records are the walk's own layout
    return dict(bytes=n * (2 * _STATE + 16 + 24.0) + g * (7 * 12.0 + 60.0),
                flops=n * case.get("intervals", 1) * case["days"] * _PER_DAY * _FLOPS_STEP + 800.0 * g)


# ---- values in 64 bits -------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _erf_diff(i, hd):
    return torch.erf((i + 0.5) / (hd * math.sqrt(2.0))) - torch.erf((i - 0.5) / (hd * math.sqrt(2.0)))


def _fold(half, nb):
    """Matrix (bin, cell) of a symmetric factor half[0..m] centred on each bin, mirrored at both grid ends."""
    m, dev = half.shape[0] - 1, half.device
    M = torch.zeros(nb, nb, dtype=torch.float64, device=dev)
    g = torch.arange(1, nb + 1, device=dev)
    for t in range(-m, m + 1):
        p = g + t
        p = torch.where(p < 1, 1 - p, p)
        p = torch.where(p > nb, 2 * nb + 1 - p, p)
        ok = p >= 1
        M[g[ok] - 1, p[ok] - 1] += half[abs(t)]
    return M


class _Database:
    """Kernels from a logarithmic table of h / bin (unit bins): spatial reconstructions."""

    def __init__(self, nb, mask, coords):
        self.nb, self.mask, self.nd, self.at, self.dev = nb, mask, sum(mask), coords, _dev()
        nd = int(math.ceil(math.log10(15.0 / 0.3) / math.log10(1.3))) + 1
        li, le = math.log10(0.3), math.log10(15.0)
        self.hod, acc = [], 0.0
        for _ in range(nd):
            self.hod.append(10.0 ** (li + acc))
            acc += (le - li) / (nd - 1)
        self.dlog = math.log(self.hod[1] / self.hod[0])
        self.memo = {}

    def level(self, h):
        i = torch.floor(torch.log(h / 0.3) / self.dlog) + 1
        i = torch.where(h <= 0, torch.ones_like(i), i)
        return torch.clamp(i, 1, len(self.hod)).long()

    def factor(self, d, lev, axis=None):
        """Folded matrix along dimension d of level lev's smoothing kernel, or (axis given) of the
        second-derivative kernel along that axis."""
        key = (d, lev, axis)
        if key not in self.memo:
            hd = self.hod[lev - 1]
            if axis is None:
                i = torch.arange(int(math.ceil(3 * hd)) + 1, dtype=torch.float64, device=self.dev)
                half = _erf_diff(i, hd)
                half = half / (half[0] + 2.0 * half[1:].sum())
            else:
                i = torch.arange(int(math.ceil(4 * hd)) + 1, dtype=torch.float64, device=self.dev)
                if d == axis:
                    c = -1.0 / (2.0 ** (self.nd - 0.5) * math.sqrt(math.pi) * hd ** 3)
                    e = [(i + s) * torch.exp(-(i + s) ** 2 / (2.0 * hd * hd)) for s in (0.5, -0.5)]
                    before = sum(self.mask[:axis])
                    half = c * (e[0] - e[1]) * hd ** (-0.5 * before)
                else:
                    half = _erf_diff(i, hd)
            self.memo[key] = _fold(half, self.nb[d])
        return self.memo[key]

    def apply(self, field, lev, axis=None, transpose=False):
        for d in range(3):
            if self.mask[d]:
                M = self.factor(d, int(lev[d]), axis)
                M = M.T if transpose else M
                field = torch.movedim(torch.tensordot(M, field, dims=([1], [2 - d])), 0, 2 - d)
        return field

    def scatter(self, values, h, axis=None):
        """Sum over the bins of value * kernel; h per dimension (smoothing) or one (second derivative)."""
        lev = torch.stack([self.level(x) for x in h]) if axis is None else self.level(h)[None].expand(3, -1)
        out = torch.zeros(self.nb[2], self.nb[1], self.nb[0], dtype=torch.float64, device=self.dev)
        key = lev[0] + 64 * (lev[1] + 64 * lev[2])
        for k in torch.unique(key).tolist():
            sel = key == k
            src = torch.zeros_like(out)
            src[self.at[2][sel], self.at[1][sel], self.at[0][sel]] = values[sel]
            out += self.apply(src, (k % 64, k // 64 % 64, k // 4096), axis, transpose=True)
        return out

    def gather(self, field, h):
        lev, out = self.level(h), torch.zeros_like(h)
        for k in torch.unique(lev).tolist():
            sel = lev == k
            out[sel] = self.apply(field, (k, k, k))[self.at[2][sel], self.at[1][sel], self.at[0][sel]]
        return out


class _ExactKernels(_Database):
    """Kernels from each bin's own smoothing: 1-D breakthrough curves of bin size b."""

    def __init__(self, nb, b, coords):
        self.nb, self.mask, self.nd, self.at, self.dev, self.b = nb, (1, 0, 0), 1, coords, _dev(), b

    def rows(self, h, axis):
        """(bin, cell) values of every bin's kernel, folded at the grid ends."""
        G, g, hd = self.nb[0], self.at[0].double()[:, None] + 1.0, (h / self.b)[:, None]
        m = torch.ceil((3.0 if axis is None else 4.0) * hd)
        q = torch.arange(1, G + 1, dtype=torch.float64, device=self.dev)[None]

        def tap(j):
            j = j.abs()
            if axis is None:
                v = 0.5 * _erf_diff(j, hd)
            else:
                e = [(j + s) * torch.exp(-(j + s) ** 2 / (2.0 * hd * hd)) for s in (0.5, -0.5)]
                v = -1.0 / (math.sqrt(2.0) * math.sqrt(math.pi) * hd ** 3) * (e[0] - e[1])
            return torch.where(j <= m, v, torch.zeros_like(v))

        R = (tap(q - g) + tap(1 - q - g)) + (tap(2 * G + 1 - q - g) + tap(q - 2 * G - g))
        if axis is None:
            k = torch.arange(0, int(m.max()) + 1, dtype=torch.float64, device=self.dev)[None]
            t = tap(k.expand(h.shape[0], -1))
            R = R / (2.0 * t.sum(1) - t[:, 0])[:, None]
        return R

    def scatter(self, values, h, axis=None):
        return (values @ self.rows(h[0] if axis is None else h, axis)).reshape(1, 1, -1)

    def gather(self, field, h):
        return self.rows(h, None) @ field.reshape(-1)


def _reconstruct(K, counts, npts, hs, size, bins, loops_max=10, rel_err=0.02):
    """The optimisation loop of GPKDE (Fernandez-Garcia and Sanchez-Vila; the reference's form) on the active
    bins: returns (density grid, loops, kernel smoothing)."""
    nd, mask, at, dev = float(K.nd), K.mask, K.at, K.dev
    dims = [d for d in range(3) if mask[d]]
    cnt = counts[at[2], at[1], at[0]]
    vol = math.prod(bins[d] for d in dims)
    max_k = {d: bins[d] * (0.9 * size[d] - 1) / 3.0 for d in dims}
    min_k = {d: 1.2 * bins[d] / 3.0 for d in dims}
    max_sd = {d: bins[d] * (0.9 * size[d] - 1) / 4.0 for d in dims}
    min_sd = {d: 1.2 * bins[d] / 4.0 for d in dims}
    sup_c = ((nd + 2) * (8 * math.pi) ** (0.5 * nd)) ** 0.25
    alpha = ((1 + 2 ** (0.5 * nd + 2)) / (3 * 2 ** (4 / (nd + 4)))) ** (1 / (nd + 6)) * (nd + 2) ** (1 / (nd + 4)) \
        / (nd + 4) ** (1 / (nd + 6))
    zero = torch.zeros_like(cnt)
    pick = lambda f: f[at[2], at[1], at[0]]  # noqa: E731

    def mean_scale(ks):
        out = torch.ones_like(cnt)
        for d in dims:
            out = out * ks[d]
        return out ** (1.0 / nd)

    def measure(nest, net, scale):
        e = (nest / (scale ** nd * (4 * math.pi) ** (0.5 * nd)) + 0.25 * net * scale ** 4) / npts ** 2
        return math.sqrt(float((torch.where(scale != 0, e, zero) ** 2).mean()))

    ks = [torch.full_like(cnt, hs) if mask[d] else zero for d in range(3)]
    scale = mean_scale(ks)
    support, shape = 2.0 * scale, [ks[d] / scale if mask[d] else zero for d in range(3)]
    dens = K.scatter(cnt, ks) / vol
    darr, net = pick(dens), zero
    alm_old = cum = cum_old = 0.0
    for m in range(1, loops_max + 1):
        darr_old, scale_old = darr, scale
        s = torch.sqrt(K.gather(dens, support)) * scale ** (1 + 0.25 * nd) / (4 * darr) ** 0.25 * sup_c
        s = torch.minimum(s, 1.5 * support)
        support = torch.clamp(s, max=min(max_k.values()))
        support = torch.clamp(support, min=max(min_k.values()))
        nest = K.gather(dens, support)
        nv = ((math.sqrt(8 * math.pi) * support) ** nd * nest * nest / darr) ** (2 / (nd + 4) / (nd + 6))
        curv = {}
        for a in dims:
            ts = sum((5.0 if k == a else 1.0) / shape[k] ** 2 for k in dims)
            h = alpha * nv * (1 / (nd + 4) / shape[a] ** 4 * ts) ** (-1 / (nd + 6)) * scale
            h = torch.clamp(h, min_sd[a], max_sd[a])
            curv[a] = K.scatter(cnt, h, a) / vol / bins[a] ** 2
        sq = {a: curv[a] ** 2 for a in dims}
        r = {a: K.gather(sq[a], support) for a in dims}
        if K.nd == 1:
            net = r[dims[0]]
        elif K.nd == 2:
            a, b = dims
            net = 2 * K.gather(curv[a] * curv[b], support) + 2 * torch.sqrt(r[a] * r[b])
        else:
            x, y, z = (r[a] for a in dims)
            net = 3 * (x * y * z) ** (1 / 3)
            for i, j, k in ((0, 1, 2), (0, 2, 1), (1, 2, 0)):  # pair (i, j), the third axis k
                c = K.gather(sq[i] * sq[j], support)
                t = 2 * c * (r[k] * r[k] / r[i] / r[j]) ** (1 / 6)
                net = net + torch.where(c > 0, t, zero)
        if K.nd > 1:
            tot = sum(r.values())
            tot = torch.where(tot == 0, net[net > 0].min(), tot)
            far = torch.stack([v / tot > 0.85 for v in r.values()]).any(0)
            net = torch.where(far, 0.5 * net + 0.5 * tot, net)
        scale = torch.where(net > 0, (nd * nest / ((4 * math.pi) ** (0.5 * nd) * net)) ** (1 / (nd + 4)), zero)
        scale = torch.where(net == 0, scale.max(), scale)
        shape = [torch.ones_like(cnt) for _ in range(3)]
        if K.nd > 1:
            ok = torch.stack([v != 0 for v in r.values()]).all(0)
            raw, p = {}, 1.0 / (8 if K.nd == 2 else 12)
            for a in dims[:-1]:
                raw[a] = torch.maximum((net / r[a]) ** p, min_k[a] / scale)
            raw[dims[-1]] = 1 / math.prod(raw.values())
            ns = torch.sqrt(math.prod(raw.values())) if K.nd == 2 else \
                math.prod(raw.values()) ** float(np.float32(0.333))
            for a in dims:
                shape[a] = torch.where(ok, raw[a] / ns, shape[a])
        new = [torch.clamp(shape[d] * scale, min_k[d], max_k[d]) if mask[d] else zero for d in range(3)]
        if any(bool((new[d] != shape[d] * scale).any()) for d in dims):
            scale = mean_scale(new)
        ks = new
        dens = K.scatter(cnt, ks) / vol
        darr = pick(dens)
        e = (darr / darr.max() - darr_old / darr_old.max()).abs() / (darr_old / darr_old.max())
        err_d = math.sqrt(float((e ** 2).mean()))
        err_s = math.sqrt(float((((scale - scale_old).abs() / scale_old) ** 2).mean()))
        alm = measure(nest, net, scale)
        cum += alm
        if (alm_old > 0 and abs(alm - alm_old) / alm_old < rel_err) or err_d < rel_err or err_s < rel_err or \
                (m > 7 and abs(cum_old / (m - 1) - cum / m) / cum_old / (m - 1) < rel_err):
            break
        alm_old, cum_old = alm, cum
    return dens, m, ks


def _exact_kde(case, seed):
    p, xyz = _plume(case, seed)
    if case["precision"] == "mixed":  # the mixed-precision handle holds its local coordinates in 32 bits
        lo = np.floor(xyz - 1e-12)
        loc = np.stack([p.lx, p.ly, p.lz], 1).astype(np.float32).astype(np.float64)
        lo[:, 0] = (p.cell - 1) % case["ncol"]
        lo[:, 1] = case["nrow"] - 1 - (p.cell - 1) // case["ncol"] % case["nrow"]
        lo[:, 2] = case["nlay"] - 1 - (p.cell - 1) // (case["ncol"] * case["nrow"])
        xyz = (1.0 - loc) * lo + loc * (lo + 1.0)
    nb = (case["ncol"], case["nrow"], case["nlay"])
    bins = np.floor(xyz).astype(np.int64)
    ok = ((bins >= 0) & (bins < np.array(nb))).all(1)
    lin = (bins[:, 0] + nb[0] * (bins[:, 1] + nb[1] * bins[:, 2]))[ok]
    mass = np.bincount(lin, weights=p.mass[ok], minlength=math.prod(nb)).reshape(nb[::-1])
    eff = float((p.mass ** 2).sum() / p.mass.sum()) if case["weighted"] else 1.0
    counts = torch.as_tensor(mass / eff, device=_dev())
    z, y, x = torch.nonzero(counts, as_tuple=True)
    mask = tuple(int(v > 1) for v in nb)
    nd, n = sum(mask), float(p.n)
    sd = [xyz[:, d].std() for d in range(3) if mask[d]]
    hs = math.prod(sd) ** (1.0 / nd) * (4.0 / ((nd + 2) * n)) ** (1.0 / (nd + 4))
    dens, loops, _ = _reconstruct(_Database(nb, mask, (x, y, z)), counts, n, hs, nb, (1.0, 1.0, 1.0))
    return [dens * eff, torch.as_tensor(mass), loops]


def _exact_series(case, seed):
    t, w = _arrivals(case, seed)
    n, q = float(t.size), t.size
    if case["bin_format"] == 0:
        b = float(np.float32(3.49)) * t.std() / n ** (1.0 / 3.0)
    else:
        s = np.sort(t)
        at = lambda i: s[i - 1]  # noqa: E731
        if q % 2 == 0:
            if q // 2 % 2 == 0:
                q1, q3 = (at(q // 4) + at(q // 4 + 1)) / 2, (at(q // 2 + q // 4) + at(q // 2 + q // 4 + 1)) / 2
            else:
                q1, q3 = at(q // 4 + 1), at(q // 2 + q // 4 + 1)
        else:
            r = (q - 1) // 4
            if (q - 1) // 2 % 2 == 0:
                q1, q3 = (at(r) + at(r + 1)) / 2, (at(q // 2 + 1 + r) + at(q // 2 + 2 + r)) / 2
            else:
                q1, q3 = at(r + 1), at(q // 2 + 2 + r)
        b = 2.0 * (q3 - q1) / n ** (1.0 / 3.0)
    b = case["fraction"] * b
    G = int(400.0 / b + 0.5)
    k = np.floor(t / b).astype(np.int64)
    ok = k < G
    fmt = case["eff_format"]
    mass = np.bincount(k[ok], weights=w[ok], minlength=G)
    eff = (w ** 2).sum() / w.sum() if fmt == 0 else 1.0
    if fmt == 0:
        counts = mass / eff
    elif fmt == 2:
        counts = np.bincount(k[ok], minlength=G).astype(np.float64)
    else:
        w2 = np.bincount(k[ok], weights=w[ok] ** 2, minlength=G)
        counts = np.where(w2 != 0, mass ** 2 / np.where(w2 != 0, w2, 1.0), 0.0)
    c = torch.as_tensor(counts, device=_dev()).reshape(1, 1, G)
    _, _, x = torch.nonzero(c, as_tuple=True)
    K = _ExactKernels((G, 1, 1), b, (x, torch.zeros_like(x), torch.zeros_like(x)))
    hs = t.std() * (4.0 / (3.0 * n)) ** 0.2
    dens, loops, ks = _reconstruct(K, c, n, hs, (G, 1, 1), (b, 1.0, 1.0))
    if fmt >= 2:
        dens = K.scatter(torch.as_tensor(mass, device=_dev())[x], ks) / b
    return [counts * eff, dens.reshape(-1) * eff, float(b), (np.arange(1, G + 1) - 0.5) * b, G, loops, int(x.numel())]


def _normals(seed, ids, step):
    """The walk's three standard normals of a step: Irwin-Hall(12) over Philox4x32-10 (Salmon et al., SC'11)."""
    M, out = 0xFFFFFFFF, []
    for d in range(3):
        tot = torch.zeros_like(ids)
        for blk in range(3):
            c = [torch.full_like(ids, 9 * step + 3 * d + blk), torch.zeros_like(ids), ids & M, ids >> 32]
            k0, k1 = seed & M, (seed >> 32) & M
            for _ in range(10):
                p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
                c = [((p1 >> 32) & M) ^ c[1] ^ k0, p1 & M, ((p0 >> 32) & M) ^ c[3] ^ k1, p0 & M]
                k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
            tot = tot + c[0] + c[1] + c[2] + c[3]
        out.append((tot - (6 << 32)).double() * 2.0 ** -32)
    return torch.stack(out, 1)


def _exact_adjoint(case, seed):
    """The differentiable walk in torch operations and its gradient by torch's own differentiation."""
    from torch.utils.checkpoint import checkpoint
    g, f, p, theta, grad = _adjoint_inputs(case, seed)
    dev, nz = _dev(), _ADJ["nz"]
    n0, n1, n2 = g.ncol, g.nrow, g.nlay
    # specific discharge through the cells' faces (+x, +y, +z), arrays over (layer, row, column)
    face = np.zeros((6, g.ncell))
    rows = np.repeat(np.arange(g.ncell), np.diff(f.ia))
    for k, (off, sgn) in enumerate(((-1, 1), (1, -1), (n0, 1), (-n0, -1), (n0 * n1, 1), (-n0 * n1, -1))):
        sel = (f.ja - 1 - rows) == off
        if n0 == 1 or abs(off) != 1:
            face[k, rows[sel]] = sgn * f.flowja[sel]
        else:
            sel &= (f.ja - 1) // n0 == rows // n0
            face[k, rows[sel]] = sgn * f.flowja[sel]
    face = face.reshape(6, n2, n1, n0)[:, ::-1, ::-1, :]  # model order: z from the bottom, y from the front
    zones = _zones(g).reshape(n2, n1, n0)[::-1, ::-1, :]
    shp = (n2 + 1, n1 + 1, n0 + 1)
    q, beta, cnt = np.zeros(shp + (3,)), np.zeros(shp + (nz,)), np.zeros(shp)
    for oz in (0, 1):
        for oy in (0, 1):
            for ox in (0, 1):
                at = (slice(oz, n2 + oz), slice(oy, n1 + oy), slice(ox, n0 + ox))
                q[at] += np.stack([face[ox], face[2 + oy], face[4 + oz]], -1)
                for z in range(nz):
                    beta[at + (z,)] += zones == z
                cnt[at] += 1.0
    q, beta = (torch.as_tensor((a / cnt[..., None]).reshape(-1, a.shape[-1]), device=dev) for a in (q, beta))
    dmr = torch.full((q.shape[0],), float(f.dm_eff[0]), dtype=torch.float64, device=dev)
    th = torch.tensor(theta, device=dev, requires_grad=True)
    aL, aT, phi = beta @ th[:nz], beta @ th[nz:2 * nz], beta @ th[2 * nz:3 * nz]
    u = th[3 * nz] * q / phi[:, None]
    eps2 = _ADJ["eps"] ** 2
    r = torch.sqrt((u * u).sum(1) + eps2)
    D = (phi * (aT * r + dmr))[:, None, None] * torch.eye(3, dtype=torch.float64, device=dev) + \
        (phi * (aL - aT) / r)[:, None, None] * u[:, :, None] * u[:, None, :]
    G = 0.0
    for j, ax in ((0, 2), (1, 1), (2, 0)):
        G = G + torch.gradient(D[:, :, j].reshape(shp + (3,)), dim=ax)[0].reshape(-1, 3)
    nodes = torch.cat([u, G / phi[:, None], aL[:, None], aT[:, None], dmr[:, None]], 1)
    L = torch.tensor([n0, n1, n2], dtype=torch.float64, device=dev)
    dt, ids = _ADJ["dt"], torch.as_tensor(p.id.astype(np.int64), device=dev)
    sdt = math.sqrt(dt)
    corners = [(x, y, z) for z in (0, 1) for y in (0, 1) for x in (0, 1)]

    def steps(x, nodes, k0, k1):
        for k in range(k0, k1):
            c = torch.minimum(torch.clamp(torch.floor(x.detach()), min=0.0), L - 1)
            fr, ci, val = torch.clamp(x - c, 0.0, 1.0), c.long(), 0.0
            for o in corners:
                w = 1.0
                for d in range(3):
                    w = w * (fr[:, d] if o[d] else 1.0 - fr[:, d])
                at = ci[:, 0] + o[0] + (n0 + 1) * (ci[:, 1] + o[1] + (n1 + 1) * (ci[:, 2] + o[2]))
                val = val + w[:, None] * nodes[at]
            v, aL, aT, dm = val[:, :3], val[:, 6], val[:, 7], val[:, 8]
            s2 = (v * v).sum(1)
            r = torch.sqrt(s2 + eps2)
            lt = aT * r + dm
            a, b = torch.sqrt(2 * lt), torch.sqrt(2 * (lt + (aL - aT) * s2 / r))
            xi = _normals(seed, ids, k)
            bxi = a[:, None] * xi + (2 * (aL - aT) / (r * (a + b)) * (v * xi).sum(1))[:, None] * v
            y = x + (v + val[:, 3:6]) * dt + bxi * sdt
            y = y - torch.floor((y / (2 * L)).detach()) * 2 * L
            x = torch.where(y > L, 2 * L - y, y)
        return x

    k = (p.cell - 1) // (n0 * n1)
    i, j = (p.cell - 1) // n0 % n1, (p.cell - 1) % n0
    x = torch.as_tensor(np.stack([j + p.lx, n1 - 1 - i + p.ly, n2 - 1 - k + p.lz], 1), device=dev)
    for k0 in range(0, case["nsteps"], 4):
        x = checkpoint(steps, x, nodes, k0, min(k0 + 4, case["nsteps"]), use_reentrant=False)
    # deposit: product biweight kernels at the bin centres
    rho = torch.zeros(n2 * n1 * n0, dtype=torch.float64, device=dev)
    c = torch.floor(x.detach()).long()
    span = [range(-int(h) - 1, int(h) + 2) for h in _ADJ["h"]]

    def factor(d, o):
        h = _ADJ["h"][d]
        t = (c[:, d] + o + 0.5 - x[:, d]) / h
        v = torch.where(t.abs() < 1.0, 15.0 / (16.0 * h) * (1.0 - t * t) ** 2, torch.zeros_like(t))
        return torch.where((c[:, d] + o >= 0) & (c[:, d] + o < L[d]), v, torch.zeros_like(v))

    fac = [{o: factor(d, o) for o in span[d]} for d in range(3)]
    for a in span[0]:
        for b in span[1]:
            for e in span[2]:
                at = (c[:, 0] + a).clamp(0, n0 - 1) + n0 * ((c[:, 1] + b).clamp(0, n1 - 1) +
                                                           n1 * (c[:, 2] + e).clamp(0, n2 - 1))
                rho = rho.index_add(0, at, fac[0][a] * fac[1][b] * fac[2][e])
    rho = rho.reshape(n2, n1, n0)
    (gth,) = torch.autograd.grad((rho * torch.as_tensor(grad, device=dev)).sum(), th)
    return [rho.detach(), gth]


def exact(case, seed):
    return {"kde": _exact_kde, "series": _exact_series, "adjoint": _exact_adjoint}.get(case["kind"],
                                                                                    lambda c, s: None)(case, seed)
