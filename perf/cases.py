"""The work that programs have this library do, as measurable cases.

Two families, each through its public entry points:

* ``sim`` / ``ensemble`` -- the ADI time step: a program holds one
  ``Simulation`` (or an ``Ensemble`` of them) on the GPU, advances it some
  steps (by replayed graph or launch by launch) and downloads the fields it
  saves, as the reference's loop does at its output times. A pass is such an
  interval; the state goes on from pass to pass.
* ``gtsv`` -- ``gtsv_batched`` on a packed batch of tridiagonal systems that is
  resident on the GPU.

The meshes run from the smallest that the tests step (64x32) to the benchmark's
2048x1024, the batches from 64 short systems to 16384 systems of up to 4096
rows, and lines of up to 16384 unknowns (a line of 8192 cells).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hydist_c_b200 as H
from hydist_c_b200 import scenario as S

PRECISION = {"fp64": H.FP64, "fp32": H.FP32, "fp32-refine": H.FP32_REFINE}
HOURS = 2000  # of boundary series: far more than the passes of a measurement advance


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a tutorial-sized channel: nothing but launches and latency
        dict(name="channel-64x32", kind="sim", N=64, M=32, dx=10.0, precision="fp64",
             sediment=False, islands=False, graph=True, steps=20),
        # the plain hydraulic configuration of the benchmark plan
        dict(name="channel-256x128", kind="sim", N=256, M=128, dx=10.0, precision="fp64",
             sediment=False, islands=False, graph=True, steps=20),
        # a mesh of the size of the reference's river data, with islands
        # (several wet segments per line), launch by launch as
        # Hydraulic_Calculation's default stepping does
        dict(name="river-464x324-eager", kind="sim", N=464, M=324, dx=10.0, precision="fp64",
             sediment=True, islands=True, graph=False, steps=20),
        # the headline workload: hydraulics, sediment and bed change
        dict(name="sediment-2048x1024", kind="sim", N=2048, M=1024, dx=5.0, precision="fp64",
             sediment=True, islands=False, graph=True, steps=20),
        # its single-precision form, saved more often
        dict(name="sediment-2048x1024-fp32", kind="sim", N=2048, M=1024, dx=5.0, precision="fp32",
             sediment=True, islands=False, graph=True, steps=10),
        # the refined form on an ensemble member's mesh, alone
        dict(name="sediment-1024x512-refine", kind="sim", N=1024, M=512, dx=5.0,
             precision="fp32-refine", sediment=True, islands=False, graph=True, steps=10),
        # scenario ensembles: a few large members, many small ones
        dict(name="ensemble-8x1024x512", kind="ensemble", members=8, N=1024, M=512, dx=5.0,
             precision="fp64", sediment=True, islands=False, graph=True, steps=10),
        dict(name="ensemble-24x256x128-fp32", kind="ensemble", members=24, N=256, M=128, dx=5.0,
             precision="fp32", sediment=True, islands=False, graph=True, steps=10),
        # one small mesh's lines: a latency-bound solve
        dict(name="gtsv-64-short", kind="gtsv", nsys=64, lo=16, hi=256, dtype="f64", refine=False),
        # the benchmark's batch, in both types
        dict(name="gtsv-16384", kind="gtsv", nsys=16384, lo=16, hi=4096, dtype="f64", refine=False),
        dict(name="gtsv-16384-f32", kind="gtsv", nsys=16384, lo=16, hi=4096, dtype="f32",
             refine=False),
        # the interleaved lines of a mesh of several thousand cells a side
        dict(name="gtsv-512-long", kind="gtsv", nsys=512, lo=4096, hi=16384, dtype="f64",
             refine=False),
    ]


def draw(rng):
    """Another case of the same ranges: any family, form, stepping and size
    (odd ones among them), no dearer than the dearest listed one."""
    logu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["sim", "sim", "ensemble", "gtsv", "gtsv"])
    if kind == "gtsv":
        if rng.random() < 0.25:
            nsys, lo, hi = logu(32, 512), logu(1024, 4096), logu(6000, 16384)
        else:
            nsys, lo = logu(64, 16384), logu(1, 64)
            hi = logu(128, 4096)
        dtype = rng.choice(["f64", "f32"])
        return dict(kind="gtsv", nsys=nsys, lo=lo, hi=hi, dtype=dtype,
                    refine=dtype == "f64" and rng.random() < 0.3)
    precision = rng.choice(["fp64", "fp64", "fp32", "fp32-refine"])
    if kind == "sim":
        c = dict(kind=kind, N=logu(64, 2048), M=logu(32, 1024))
    else:
        c = dict(kind=kind, members=rng.randint(2, 24), N=logu(64, 512), M=logu(32, 256))
    c["M"] = min(c["M"], c["N"])  # (the reference's y sweep writes columns up to N only)
    c.update(dx=rng.choice([5.0, 10.0]), precision=precision, sediment=rng.random() < 0.7,
             islands=rng.random() < 0.3, graph=kind == "ensemble" or rng.random() < 0.7,
             steps=rng.randint(8, 20) if precision == "fp64" else rng.randint(4, 10))
    return c


# ------------------------------------------------------------------- inputs
def bundle(case, seed):
    """A channel scenario: sloping bed with bumps, banks along both sides, a
    discharge inflow and a tidal outflow, long waves of a decimetre in the
    initial level (so that the whole mesh moves from the first step), a
    concentration that varies along the channel, Fw in the range of the
    reference's own map; with islands, dry ellipses in mid-channel."""
    N, M, dx = case["N"], case["M"], case["dx"]
    rng = np.random.default_rng(seed)
    b = S.make_channel(N=N, M=M, seed=int(rng.integers(1 << 30)), dx=dx, dt=2.0, hours=HOURS,
                       inflow=float(rng.uniform(0.4, 0.8)) * M * dx,
                       tide_amp=float(rng.uniform(0.2, 0.5)), fw=(0.005, 0.0755),
                       sediment=case["sediment"], sediment_start=0.0, n_bumps=0)
    sc = b["scenario"]
    i = np.arange(N + 3, dtype=np.float64)[:, None]
    j = np.arange(M + 3, dtype=np.float64)[None, :]
    bed = 2.0 * np.ones((N + 3, M + 3))
    for _ in range(8):
        s = rng.uniform(0.04, 0.15) * min(N, M)
        gi = np.exp(-((i - rng.uniform(2, N)) / s) ** 2 / 2)
        gj = np.exp(-((j - rng.uniform(2, M)) / s) ** 2 / 2)
        bed += rng.uniform(-0.8, 0.8) * gi * gj
    sc["h"] = np.where(sc["h"] > 0, np.maximum(sc["h"] + bed, 2.0), 0.0)
    z0 = np.zeros((N + 3, M + 3))
    for _ in range(3):
        ki, kj = rng.uniform(-1, 1, 2) * 2 * np.pi / np.array([max(N / 6, 32), max(M / 4, 32)])
        ph = rng.uniform(0, 2 * np.pi)
        z0 += rng.uniform(0.02, 0.08) * (np.cos(ki * i) * np.cos(kj * j + ph) -
                                         np.sin(ki * i) * np.sin(kj * j + ph))
    sc["z0"] = z0
    if case["sediment"]:
        sc["FS0"] = sc["FS0"] * (1 + 0.4 * np.sin(6 * np.pi * i / N) * np.cos(2 * np.pi * j / M))
        b["options"]["bed_change"] = 1
    if case["islands"]:
        for q in range(6):
            ci, cj = N * (q + 1) / 7.0, M * rng.uniform(0.25, 0.75)
            ri, rj = max(2.0, N * rng.uniform(0.02, 0.05)), max(2.0, M * rng.uniform(0.04, 0.1))
            sc["h"] = np.where(((i - ci) / ri) ** 2 + ((j - cj) / rj) ** 2 < 1, 0.0, sc["h"])
    return b


def fields(case):
    """What the reference saves, and in FP64 the bed change (a small difference
    of fluxes, of which the single-precision forms keep four digits)."""
    if not case["sediment"]:
        return ["u", "v", "z"]
    return ["u", "v", "z", "FS", "dH"] if case["precision"] == "fp64" else ["u", "v", "z", "FS"]


def systems(case, seed):
    """A packed diagonally dominant batch: lengths log-uniform in [lo, hi] (a
    mesh's wet segments: the same from seed to seed), the values from the seed."""
    rng = np.random.default_rng(case["nsys"])
    n = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"] + 1), case["nsys"])).astype(np.int32)
    return S.tridiag_batch(seed=seed, lengths=n)


class State:
    """What the program holds between passes."""


def prepare(case, seed):
    st = State()
    st.case = case
    if case["kind"] == "gtsv":
        *rows, off, ln = systems(case, seed)
        t = torch.float64 if case["dtype"] == "f64" else torch.float32
        st.rows = [torch.from_numpy(a).cuda().to(t) for a in rows]
        st.off, st.ln = torch.from_numpy(off).cuda(), torch.from_numpy(ln).cuda()
        st.x = torch.empty_like(st.rows[1])
        return st
    count = case["members"] if case["kind"] == "ensemble" else 1
    prec = PRECISION[case["precision"]]
    st.sims = [H.Simulation(bundle(case, seed * 64 + k), precision=prec) for k in range(count)]
    st.ens = H.Ensemble(st.sims) if case["kind"] == "ensemble" else None
    # pinned buffers for the saved fields, as a program that saves often keeps
    shape = (case["N"] + 3, case["M"] + 3)
    st.out = [{f: torch.empty(shape, dtype=torch.float64).pin_memory().numpy()
               for f in fields(case)} for _ in st.sims]
    return st


def run(st):
    c = st.case
    if c["kind"] == "gtsv":
        return H.gtsv_batched(*st.rows, st.off, st.ln, x=st.x, refine=c["refine"])
    if st.ens is not None:
        st.ens.step(c["steps"])
    elif c["graph"]:
        st.sims[0].step_graph(c["steps"])
    else:
        st.sims[0].step(c["steps"])
    saved = [{f: s.download(f, out=o[f]) for f in fields(c)} for s, o in zip(st.sims, st.out)]
    if c["precision"] != "fp64":  # the single-precision forms' fields are kept as such
        saved = [{f: torch.from_numpy(a).float() for f, a in d.items()} for d in saved]
    # (an ensemble's fields stacked member by member would be another copy)
    return saved[0] if st.ens is None else {f: [d[f] for d in saved] for f in ("u", "z")}


def work(case):
    """A batched solve reads four arrays and writes one, 8 flops per unknown.
    A step cannot do without its carried state once in and out and its static
    fields once in: 21 values per cell in the hydraulic step, 29 with sediment
    and bed change (3 and 4 fewer of them in FP32, halved but for the FP64
    water level); about 400 flops per cell, 700 with sediment. Each saved
    field crosses once."""
    if case["kind"] == "gtsv":
        n = sum(len(a) for a in systems(case, 1)[:1])
        return dict(bytes=n * (40 if case["dtype"] == "f64" else 20), flops=8 * n)
    cells = case["N"] * case["M"] * case.get("members", 1)
    per = {("fp64", False): 168, ("fp64", True): 232}.get(
        (case["precision"], case["sediment"]), 152 if case["sediment"] else 112)
    return dict(bytes=cells * (per * case["steps"] + 8 * len(fields(case))),
                flops=cells * case["steps"] * (700 if case["sediment"] else 400))


# --------------------------------------------- the same in 64 bits, plainly
def exact(case, seed):
    """What run() returns for a new state: the batch by serial elimination in
    each system (all systems side by side), the time step restated for the
    island-free channel of bundle() (one wet segment per line, nothing
    dries); None with islands."""
    if case["kind"] == "gtsv":
        dt = np.float64 if case["dtype"] == "f64" else np.float32
        *rows, off, ln = systems(case, seed)
        return torch.from_numpy(_thomas(*(a.astype(dt).astype(np.float64) for a in rows), off, ln))
    if case["islands"]:
        return None
    if case["kind"] == "ensemble":
        got = [_Channel(bundle(case, seed * 64 + k)).run(case["steps"], ("u", "z"))
               for k in range(case["members"])]
        return {f: [d[f] for d in got] for f in ("u", "z")}
    return _Channel(bundle(case, seed * 64)).run(case["steps"], fields(case))


def _thomas(a, d, c, b, off, ln):
    order = np.argsort(-ln, kind="stable")
    off, ln = off[order].astype(np.int64), ln[order]
    active = [int(np.searchsorted(-ln, -k, side="left")) for k in range(int(ln.max()) + 1)]
    w, x = np.zeros_like(d), np.zeros_like(d)  # active[k]: systems longer than k
    o = off[:active[0]]
    w[o], x[o] = c[o] / d[o], b[o] / d[o]
    for k in range(1, int(ln.max())):
        q = off[:active[k]] + k
        m = d[q] - a[q] * w[q - 1]
        w[q], x[q] = c[q] / m, (b[q] - a[q] * x[q - 1]) / m
    for k in range(int(ln.max()) - 2, -1, -1):
        q = off[:active[k + 1]] + k
        x[q] -= w[q] * x[q + 1]
    return x


class _Channel:
    """The ADI step of an island-free channel (wet rows 2..N, columns
    3..M-1; discharge on the left, level on the right, solid sides), in the
    reference's order of operations on whole arrays. A direction's arrays are
    passed along x cross: transposed for the y half-step, whose formulas are
    the x half-step's with the velocities exchanged."""

    def __init__(self, b):
        sc, self.p = b["scenario"], H.capi.params_from_dict(b["params"])
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        self.N, self.M, p = sc["N"], sc["M"], self.p
        N, M, h, n = self.N, self.M, t(sc["h"]), t(sc["hsnham"])
        self.h, self.vis, self.Fw = h, t(sc["visco"]), t(sc["Fw"])
        zero = lambda: torch.zeros_like(h)  # noqa: E731
        self.ht, self.Kx1, self.Ky1 = zero(), zero(), zero()
        self.wet = torch.zeros_like(h, dtype=torch.bool)
        mean = (h[:-1, :-1] + h[:-1, 1:] + h[1:, :-1] + h[1:, 1:]) * 0.25
        self.ht[1:N + 1, 1:M + 1] = mean[:N, :M]
        self.wet[1:N + 2, 1:M + 2] = mean[:N + 1, :M + 1] > 0
        for K, ha, na in ((self.Kx1, h[:, :-1] + h[:, 1:], n[:, :-1] + n[:, 1:]),
                          (self.Ky1, h[:-1] + h[1:], n[:-1] + n[1:])):
            k = torch.where(ha != 0, p.g * (ha * 0.5).clamp(min=1e-300) ** (-2 * p.mu_mn) * (na * 0.5) ** 2, 0.0)
            K[1:N + 1, 1:M + 1] = k[1:N + 1, :M] if K is self.Kx1 else k[:N, 1:M + 1]
        self.u, self.v, self.tu, self.tv, self.Hm = zero(), zero(), zero(), zero(), zero()
        self.z, self.tz = t(sc["z0"]), t(sc["z0"])
        self.Hu, self.Hv, self.VTH, self.Kx, self.Ky, self.dH = (zero() for _ in range(6))
        self.depths()
        self.sed = sc["FS0"] is not None
        self.FS = t(sc["FS0"]) if self.sed else zero()
        self.tFS = self.FS.clone()
        wl = (h[1, 3:M] + h[1, 2:M - 1]) / 2  # the inflow's weights
        self.weight = wl ** (2 / 3) / ((wl ** (5 / 3)).sum() * p.dX)
        self.q, self.right, self.cin = sc["bc_left"], sc["bc_right"], sc["CC_left"]
        self.hmax = 1 / (p.ros * float(self.ht[2, 2:M].max()))
        self.t = 0.0

    def depths(self):
        N, M, h, z = self.N, self.M, self.h, self.z
        i, j = slice(1, N + 1), slice(1, M + 1)
        self.Hu[i, j] = (h[i, :M] + h[i, j] + z[2:N + 2, j] + z[i, j]) * 0.5
        self.Hv[i, j] = (h[:N, j] + h[i, j] + z[i, 2:M + 2] + z[i, j]) * 0.5

    def boundary(self):
        self.t += self.p.dT / 2
        k, M, N = int(self.t // 3600), self.M, self.N
        w = self.t / 3600 - k
        at = lambda s: s[k] * (1 - w) + s[k + 1] * w  # noqa: E731
        self.ub = at(self.q) * self.weight
        self.tz[N:N + 2, 3:M] = at(self.right)
        self.FS[2, 3:M] = at(self.cin) * self.ht[2, 3:M] * self.hmax

    def cross(self, b, A, lim, dry_lo, dry_hi, dry_lo2, m2, m1, p1, p2):
        """First and second difference of A along an axis, one-sided (and only
        upwind) beside dry cells."""
        first = torch.where(dry_lo, torch.where(b < 0, -3 * A + 4 * p1 - p2, 0.0),
                            torch.where(dry_hi, torch.where(~dry_lo2 & (b > 0), 3 * A - 4 * m1 + m2, 0.0), p1 - m1))
        second = torch.where(dry_lo, torch.where(b < 0, A - 2 * p1 + p2, 0.0),
                             torch.where(dry_hi, torch.where(~dry_lo2 & (b > 0), A - 2 * m1 + m2, 0.0), p1 - 2 * A + m1))
        return first * lim, second

    def sweep(self, a, b, ta, Ha, Hb, K, tr):
        """The implicit half-step of the velocity `a` along the lines and the
        level, by the continuity rows put into the momentum rows."""
        p, d = self.p, self.p.dX
        f = lambda x: x.t() if tr else x  # noqa: E731
        a, b, ta, Ha, Hb, K, vis, Hm, z, tz = (f(x) for x in (a, b, ta, Ha, Hb, K, self.vis, self.Hm, self.z, self.tz))
        first, last = (3, self.M - 1) if tr else (2, self.N)
        P, l0, l1 = slice(first, last + 1), (2 if tr else 3), (self.N if tr else self.M - 1)
        L = slice(l0, l1 + 1)
        sh = lambda X, o, c: X[first + o:last + 1 + o, l0 + c:l1 + 1 + c]  # noqa: E731
        k, f4 = p.dT / (2 * d), 2 * p.g * p.dT / (2 * d)
        bb = (sh(b, 0, -1) + sh(b, 0, 0) + sh(b, 1, -1) + sh(b, 1, 0)) * 0.25
        A, VI, rH = sh(a, 0, 0), sh(vis, 0, 0), 1 / sh(Ha, 0, 0)
        visc = VI * p.dT / (d * d)
        f1, f3 = k * A + visc, visc - k * A
        f2 = -(2 + sh(K, 0, 0) * p.dT * torch.sqrt(A * A + bb * bb) * rH + 2 * visc)
        dry = lambda c: sh(Hm, 0, c) <= p.H_TINH  # noqa: E731
        adv, lap = self.cross(bb, A, bb / (2 * d), dry(-1), dry(1), dry(-2), sh(a, 0, -2), sh(a, 0, -1),
                              sh(a, 0, 1), sh(a, 0, 2))
        f5 = -2 * A + p.dT * adv - p.dT * VI * lap / (d * d)
        c2, a2 = k * sh(Ha, 0, 0), -k * sh(Ha, -1, 0)
        d2 = sh(z, 0, 0) - k * (sh(Hb, 0, 0) * sh(b, 0, 0) - sh(Hb, 0, -1) * sh(b, 0, -1))
        LO, DI = f1 - f4 * a2, f2[:-1] - f4 * (c2[:-1] - a2[1:])
        UP, RH = f3[:-1] + f4 * c2[1:], f5[:-1] + f4 * (d2[1:] - d2[:-1])
        if not tr:  # inflow at the first end; no velocity beyond the last
            RH[0] -= LO[0] * self.ub
        m = last - first
        w, x = torch.empty_like(UP), torch.empty_like(RH)
        w[0], x[0] = UP[0] / DI[0], RH[0] / DI[0]
        for i in range(1, m):
            q = 1 / (DI[i] - LO[i] * w[i - 1])
            w[i], x[i] = UP[i] * q, (RH[i] - LO[i] * x[i - 1]) * q
        for i in range(m - 2, -1, -1):
            x[i] -= w[i] * x[i + 1]
        lo = torch.zeros_like(x[:1]) if tr else self.ub[None]
        prev = torch.cat([lo, x])
        zz = d2 - a2 * prev
        zz[:-1] -= c2[:-1] * x
        ta[first:last, L] = x
        ta[first - 1, L] = lo[0]
        tz[first:last, L] = zz[:-1]
        if tr:
            ta[last, L], tz[last, L] = 0.0, zz[-1]
        else:
            ta[last, L] = (d2[-1] - a2[-1] * x[-1] - tz[last, L]) / c2[-1]

    def smooth(self, x, along):
        """The smoothed velocity: its two neighbours along its own direction
        and, where wet, the two across."""
        N, M, p = self.N, self.M, self.p
        I, J = slice(2, N + 1), slice(2, M + 1)
        up, dn, le, ri = x[1:N, J], x[3:N + 2, J], x[I, 1:M], x[I, 3:M + 2]
        w = self.wet
        wu, wd, wl, wr = w[1:N, J], w[3:N + 2, J], w[I, 1:M], w[I, 3:M + 2]
        if along == 0:
            nb, n = up + dn + torch.where(wl, le, 0.0) + torch.where(wr, ri, 0.0), 2 + wl.double() + wr.double()
        else:
            nb, n = le + ri + torch.where(wu, up, 0.0) + torch.where(wd, dn, 0.0), 2 + wu.double() + wd.double()
        out = x.clone()
        out[I, J] = torch.where(x[I, J] != 0, x[I, J] * p.heso + (1 - p.heso) * nb / n, x[I, J])
        return out

    def explicit(self, a, b, sb, ta, Ha, K, tr):
        """The explicit half-step of the velocity `a` across the lines; in the
        layout along x cross, a's own direction is the second axis."""
        p, d = self.p, self.p.dX
        f = lambda x: x.t() if tr else x  # noqa: E731
        a, b, sb, ta, Ha, K, vis, Hm, z = (f(x) for x in (a, b, sb, ta, Ha, K, self.vis, self.Hm, self.z))
        p0, p1 = (3, self.M) if tr else (2, self.N + 1)
        l0, l1 = (1, self.N) if tr else (3, self.M - 1)
        sh = lambda X, o, c: X[p0 + o:p1 + o, l0 + c:l1 + c]  # noqa: E731
        mean = lambda X: (sh(X, -1, 0) + sh(X, 0, 0) + sh(X, -1, 1) + sh(X, 0, 1)) * 0.25  # noqa: E731
        bb, tb, A, rH = mean(b), mean(sb), sh(a, 0, 0), 1 / sh(Ha, 0, 0)
        dry = lambda o: sh(Hm, o, 0) <= p.H_TINH  # noqa: E731
        q, lap = self.cross(bb, A, tb / (2 * d), dry(-1), dry(1), dry(-2), sh(a, -2, 0), sh(a, -1, 0),
                            sh(a, 1, 0), sh(a, 2, 0))
        den = 2 / p.dT + (sh(a, 0, 1) - sh(a, 0, -1)) / (2 * d) + sh(K, 0, 0) * torch.sqrt(bb * bb + A * A) * rH
        num = (2 / p.dT * A - q - p.g * (sh(z, 0, 1) - sh(z, 0, 0)) / d +
               sh(vis, 0, 0) * (lap + sh(a, 0, 1) - 2 * A + sh(a, 0, -1)) / (d * d))
        ta[p0:p1, l0:l1] = num / den

    def commit(self):
        N, M, i, j = self.N, self.M, slice(0, self.N + 1), slice(0, self.M + 1)
        self.u[i, j], self.v[i, j], self.z[i, j] = self.tu[i, j], self.tv[i, j], self.tz[i, j]
        w = self.wet[1:N + 1, 1:M + 1]
        self.Hm[1:N + 1, 1:M + 1] = torch.where(w, (self.ht + self.tz)[1:N + 1, 1:M + 1], self.Hm[1:N + 1, 1:M + 1])
        self.depths()

    def speeds(self, hi):
        """Speed and diffusivities on rows up to hi, from the committed state."""
        p, N, M, h = self.p, self.N, self.M, self.h
        i, j = slice(2, hi + 1), slice(2, M + 1)
        ut, vt = (self.tu[i, j] + self.tu[1:hi, j]) * 0.5, (self.tv[i, j] + self.tv[i, 1:M]) * 0.5
        wet = (self.ht[i, j] > 0) & (self.Hm[i, j] > p.H_TINH)
        self.VTH[i, j] = torch.where(wet, torch.sqrt(ut * ut + vt * vt), 0.0)
        i, j, ks = slice(1, hi + 1), slice(1, M + 1), 2.5 * p.dm
        for K, Hd, hs, t in ((self.Kx, self.Hu, h[i, :M] + h[i, j], self.tu), (self.Ky, self.Hv, h[:hi, j] + h[i, j], self.tv)):
            cz = 18 * torch.log(12 * Hd[i, j].clamp(min=1e-300) / ks)
            k = 5.93 * math.sqrt(p.g) * hs * 0.25 * t[i, j].abs() / cz
            K[i, j] = torch.where(Hd[i, j] > 0, k.clamp(5, 100), K[i, j])

    def ends(self):
        """The concentration of the open rows, interpolated along the flow."""
        p, N, M = self.p, self.N, self.M
        j = slice(1, M)
        for loc in (N, 2):
            t = self.tu[loc, j]
            dx = (self.u[loc, j] + t) * 0.25 * p.dT
            i = torch.trunc((N - 1 if loc == N else 2) + (-1 if loc == N else 1) * dx / p.dX).long().clamp(0, N + 1)
            F = self.FS[:, j]
            lo, hi = F.gather(0, i[None])[0], F.gather(0, i[None] + 1)[0]
            s = -1 if loc == N else 1
            whole = torch.trunc(torch.round(dx) / round(p.dX))
            self.FS[loc, j] = torch.where(t > 0, lo + s * (hi - lo) * (dx / p.dX - whole), self.FS[loc, j])

    def source(self, P, fs, vth, Hm, cut):
        p = self.p
        cc = 18 * torch.log(12 * Hm / (2.5 * p.dm))
        uf, om = math.sqrt(p.g) * vth.abs() / cc, 1 - fs
        ws = p.wss * om ** 4
        zf = torch.where(fs > cut, ws / (0.4 * (uf + 2 * ws)), 0.0)
        tob = p.ro * self.Fw[P] * vth * vth
        toe = torch.where(Hm > p.ghtoe, p.Toe * (1 + p.hstoe * (Hm - p.ghtoe)), torch.full_like(Hm, p.Toe))
        pd = (1 - tob / p.Tod).clamp(min=0)
        settle = -ws * (1 + zf / (1.25 + 4.75 * pd ** 2.5)) * fs * pd
        return torch.where(tob > toe, p.Mbochat / p.ros * (tob - toe) / toe, torch.where(tob < p.Tod, settle, 0.0)), zf

    def concentration(self, tr):
        p, d, N, M = self.p, self.p.dX, self.N, self.M
        f = lambda x: x.t() if tr else x  # noqa: E731
        f0, f1 = (4, M - 2) if tr else (3, N - 1)
        l0, l1 = (3, N - 1) if tr else (3, M - 1)
        P = (slice(l0, l1 + 1), slice(f0, f1 + 1)) if tr else (slice(f0, f1 + 1), slice(l0, l1 + 1))
        FS, tFS, Hm = f(self.FS), f(self.tFS), f(self.Hm)
        va, ha, ka = (f(x) for x in ((self.tv, self.Hv, self.Ky) if tr else (self.tu, self.Hu, self.Kx)))
        vb, hb, kb = (f(x) for x in ((self.tu, self.Hu, self.Kx) if tr else (self.tv, self.Hv, self.Ky)))
        sh = lambda X, o, c: X[f0 + o:f1 + 1 + o, l0 + c:l1 + 1 + c]  # noqa: E731
        fs, Hc = sh(FS, 0, 0), sh(Hm, 0, 0)
        src, zf = self.source(P, self.FS[P], self.VTH[P], self.Hm[P], 1e-5)
        src, zf = f(src), f(zf)
        gam = 0.98 - 0.198 * zf + 0.032 * zf * zf if tr else torch.full_like(fs, 0.98)
        r, hk, hkm = 1 / (d * d * Hc), sh(ha, 0, 0) * sh(ka, 0, 0), sh(ha, -1, 0) * sh(ka, -1, 0)
        adv = gam * 0.5 * (sh(va, 0, 0) + sh(va, -1, 0)) / (2 * d)
        A, C, B = -adv - hkm * r, adv - hk * r, 2 / p.dT + (hk + hkm) * r
        wet = lambda c: sh(Hm, 0, c) > p.H_TINH  # noqa: E731
        fp, fm = sh(FS, 0, 1), sh(FS, 0, -1)
        diff = r * (sh(hb, 0, 0) * sh(kb, 0, 0) * torch.where(wet(-1) & wet(2), fp - fs, 0.0) -
                    sh(hb, 0, -1) * sh(kb, 0, -1) * torch.where(wet(-2) & wet(1), fs - fm, 0.0))
        q = torch.where(wet(-2) & wet(2), (sh(vb, 0, 0) + sh(vb, 0, -1)) * 0.5 * (fp - fm) / (2 * d) * gam, 0.0)
        D = fs * 2 / p.dT - q + diff + src / Hc
        a0, a1, L = f0 - 1, f1 + 1, slice(l0, l1 + 1)
        for at, row, X in ((a0, 0, A), (a1, -1, C)):
            solid = torch.ones_like(B[0], dtype=torch.bool) if tr else va[at, L] == 0
            if not tr and at == a1:
                solid = torch.zeros_like(solid)  # (the i-sweep asks for a solid end as well)
            B[row] += torch.where(solid, X[row], 0.0)
            D[row] -= torch.where(solid, 0.0, X[row] * FS[at, L])
        w, x, m = torch.empty_like(C), torch.empty_like(D), f1 - f0 + 1
        w[0], x[0] = C[0] / B[0], D[0] / B[0]
        for i in range(1, m):
            g = 1 / (B[i] - A[i] * w[i - 1])
            w[i], x[i] = C[i] * g, (D[i] - A[i] * x[i - 1]) * g
        for i in range(m - 2, -1, -1):
            x[i] -= w[i] * x[i + 1]
        tFS[f0:f1 + 1, L] = torch.where(x < 0, torch.full_like(x, p.NDnen), x)
        for at, nx in ((a0, f0), (a1, f1)):
            solid = torch.ones_like(B[0], dtype=torch.bool) if tr else va[at, L] == 0
            tFS[at, L] = torch.where(solid, tFS[nx, L], FS[at, L])
        self.FS[1:N + 1, 1:M + 1] = self.tFS[1:N + 1, 1:M + 1]

    def bed(self, vth, Hm):
        """The bed-load flux of the second commit and the bed change."""
        p, d, N, M, ks = self.p, self.p.dX, self.N, self.M, 2.5 * self.p.dm
        P = (slice(2, N + 1), slice(2, M + 1))
        toe = torch.where(Hm[P] > p.ghtoe, p.Toe * (1 + p.hstoe * (Hm[P] - p.ghtoe)), torch.full_like(Hm[P], p.Toe))
        tx = (p.ro * self.Fw[P] * vth[P] ** 2 / toe - 1).clamp(min=0)
        base = (0.053 * math.sqrt((p.Sx - 1) * p.g) * p.dm ** 1.5 * tx ** 2.1 *
                (p.dm * (p.g * (p.Sx - 1) / p.muy * p.muy) ** (1 / 3)) ** -0.3)
        on = (vth[P] != 0) & self.wet[P]
        pad = lambda x: torch.nn.functional.pad(x[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]  # noqa: E731
        qx = pad(torch.where(on, base * (self.tu[P] + self.tu[1:N, 2:M + 1]) * 0.5 / vth[P], 0.0))
        qy = pad(torch.where(on, base * (self.tv[P] + self.tv[2:N + 1, 1:M]) * 0.5 / vth[P], 0.0))
        P, FS = (slice(3, N - 1), slice(3, M)), self.FS  # qx, qy start at row and column 1
        t = (qx[3:N - 1, 2:M - 1] - qx[1:N - 3, 2:M - 1]) / (2 * d) + (qy[2:N - 2, 3:M] - qy[2:N - 2, 1:M - 2]) / (2 * d)
        hkx, hky = self.Hu * self.Kx, self.Hv * self.Ky
        i, j = P
        t = t + (hkx[i, j] * (FS[4:N, j] - FS[i, j]) - hkx[2:N - 2, j] * (FS[i, j] - FS[2:N - 2, j])) / (d * d)
        t = t + (hky[i, j] * (FS[i, 4:M + 1] - FS[i, j]) - hky[i, 2:M - 1] * (FS[i, j] - FS[i, 2:M - 1])) / (d * d)
        src, _ = self.source(P, FS[P], vth[P], Hm[P], 0.0)
        self.dH[P] += p.dT / (1 - p.Dorong) * (src + t)

    def run(self, steps, names):
        for _ in range(steps):
            for tr in (False, True):
                self.boundary()
                a, b, ta, tb = (self.v, self.u, self.tv, self.tu) if tr else (self.u, self.v, self.tu, self.tv)
                Ha, Hb, Ka, Kb = (self.Hv, self.Hu, self.Ky1, self.Kx1) if tr else (self.Hu, self.Hv, self.Kx1, self.Ky1)
                self.sweep(a, b, ta, Ha, Hb, Ka, tr)
                sa = self.smooth(ta, 1 if tr else 0)
                self.explicit(b, a, sa, tb, Hb, Kb, tr)
                if tr:
                    tb[1, 3:self.M] = 2 * tb[2, 3:self.M] - tb[3, 3:self.M]
                    tb[self.N, 3:self.M] = 2 * tb[self.N - 1, 3:self.M] - tb[self.N - 2, 3:self.M]
                else:
                    tb[2:self.N + 1, 2], tb[2:self.N + 1, self.M - 1] = 0.0, 0.0
                sb = self.smooth(tb, 0 if tr else 1)
                i, j = slice(0, self.N + 1), slice(0, self.M + 1)
                ta[i, j], tb[i, j] = sa[i, j], sb[i, j]
                self.commit()
                if self.sed:
                    self.speeds(self.N - 1 if tr else self.N)
                    self.ends()
                    self.concentration(tr)
                    if tr:
                        self.bed(self.VTH, self.Hm)
        return {f: getattr(self, f).cpu() for f in names}
