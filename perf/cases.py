"""The work that a user of this library has it do, as cases that can be timed and checked.

Four kinds of call, each through the public entry points (include/c3d_b200.h, c3d.py):

  step     SSP-RK2 time steps of one problem: state in, c3d_step, state out. M_N problems start
           from a gaussian pulse over a floor (the first steps of a run) or from a transported
           field whose warm starts lag the moments (the middle of a run, where every cell needs
           Newton steps); FP64 or mixed closure, Gaunt or direct Hessian. P_N problems take the
           moment flux or the kinetic flux.
  vectors  standalone closure of independent moment vectors of the orders 1..N in one launch.
  serve    one pass of a server: a step of each of several problems in one launch.
  flux     the host-to-host kinetic flux that a build of the reference code links.
  hessian  the host-to-host Hessian batch that such a build links.

Newton tolerance 1e-6 throughout, as the repository's benchmark decks: at 1e-8 the stopping
rules of the reference are decided by single rounding errors on these problems.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("c3d-2015_b200"))
import c3d  # noqa: E402

TOL = 1e-6
LADDER = (0.0, 1e-8, 1e-6, 1e-4, 1e-2, 1e-1)
THETA = 2.0
CFL = 0.5


def listed():
    pulse = dict(kind="step", solver="mn", field="pulse", precision="fp64", hessian="gaunt",
                 sigma_s=1.0, checker=0)
    aged = dict(kind="step", solver="mn", field="aged", precision="fp64", hessian="gaunt",
                sigma_s=10.0, checker=0)
    return [
        # the smallest deck of the repository (M_2 on 16^3), where launches count
        dict(pulse, name="m2 16 fp64", N=2, Q=12, nx=16, ny=16, nz=16, width=0.1, floor=1e-4,
             steps=2),
        # the M_4 drop-in deck with the scattering checkerboard
        dict(pulse, name="m4 64 checker fp64", N=4, Q=20, nx=64, ny=64, nz=64, width=0.05,
             floor=1e-6, checker=8, steps=2),
        # a drop-in M_3 run on a grid whose edges divide by nothing
        dict(pulse, name="m3 odd fp64", N=3, Q=14, nx=37, ny=45, nz=51, width=0.15, floor=1e-8,
             steps=2),
        # M_6 near the realizability boundary in FP64, and the largest problem: the benchmark's
        # grid in mixed precision
        dict(pulse, name="m6 64 fp64", N=6, Q=28, nx=64, ny=64, nz=64, width=0.02, floor=1e-10,
             steps=2),
        dict(pulse, name="m6 128 mixed", N=6, Q=28, nx=128, ny=128, nz=128, width=0.02,
             floor=1e-10, precision="mixed", steps=2),
        # the middle of a run: every cell needs several Newton iterations
        dict(aged, name="m3 aged 48 fp64", N=3, Q=12, nx=48, ny=48, nz=48, steps=1),
        dict(aged, name="m5 aged mixed", N=5, Q=16, nx=40, ny=36, nz=44, precision="mixed",
             steps=1),
        # standalone closures, all orders in one launch
        dict(kind="vectors", name="vectors fp64", N=7, n=8192, precision="fp64", smax=1.0),
        dict(kind="vectors", name="vectors mixed", N=7, n=8192, precision="mixed", smax=1.0),
        # a pass of the serving loop: six problems, orders 1, 3 and 5
        dict(kind="serve", name="serve 6", count=6, lo=16, hi=40, precision="fp64"),
        # the linear solver
        dict(kind="step", name="p5 64", solver="pn", field="pulse", precision="fp64",
             hessian="gaunt", sigma_s=1.0, checker=0, N=5, Q=12, nx=64, ny=64, nz=64, width=0.2,
             floor=1e-4, steps=2),
        # what a build of the reference code calls: Hessians of a batch from host buffers
        dict(kind="hessian", name="hessians m6 host", N=6, Q=28, n=500, form="sparse"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["pulse", "pulse", "pulse", "aged", "aged", "vectors", "serve", "pn",
                       "flux", "hessian"])
    N = rng.randint(1, 6)
    Q = rng.choice([2 * (N + 3), 2 * (N + 3), 4 * N + 4])
    top = 64 if N >= 5 else 80
    edges = [_log_int(rng, 12, top) for _ in range(3)]
    if rng.random() < 0.5:  # cubes and even edges are the usual thing
        edges = [2 * (edges[0] // 2)] * 3
    precision = rng.choice(["fp64", "fp64", "mixed"])
    hessian = "gaunt" if precision == "mixed" or rng.random() < 0.85 else "direct"
    c = dict(kind="step", solver="mn", N=N, Q=Q, nx=edges[0], ny=edges[1], nz=edges[2],
             precision=precision, hessian=hessian, sigma_s=round(rng.uniform(0.5, 20.0), 3),
             checker=0)
    if what == "pulse":
        return dict(c, field="pulse", width=round(rng.uniform(0.03, 0.2), 4),
                    floor=10.0 ** rng.randint(-9, -4), steps=rng.randint(1, 3),
                    checker=rng.choice([0, 0, 8]))
    if what == "aged":
        # bounded cost: every cell takes several Hessians
        e = [max(8, min(v, 48 if N <= 3 else 36)) for v in edges]
        return dict(c, field="aged", nx=e[0], ny=e[1], nz=e[2], steps=1)
    if what == "vectors":
        return dict(kind="vectors", N=rng.randint(1, 7), n=_log_int(rng, 64, 12000),
                    precision=precision, smax=round(rng.uniform(0.3, 1.0), 3))
    if what == "serve":
        lo = rng.randint(12, 20)
        return dict(kind="serve", count=rng.randint(2, 8), lo=lo, hi=rng.randint(lo + 4, 40),
                    precision=precision)
    if what == "pn":
        return dict(c, solver="pn", field="pulse", precision="fp64", hessian="gaunt",
                    flux=rng.choice(["moment", "moment", "kinetic"]), Q=2 * (N + 1),
                    width=round(rng.uniform(0.1, 0.3), 4), floor=1e-4, steps=rng.randint(1, 4))
    if what == "flux":
        return dict(kind="flux", N=min(N, 5), Q=2 * (min(N, 5) + 3), nx=min(edges[0], 40),
                    ny=min(edges[1], 40), nz=min(edges[2], 40))
    return dict(kind="hessian", N=N, Q=Q, n=_log_int(rng, 10, 1000),
                form=rng.choice(["direct", "sparse", "sparse"]))


# ---------------------------------------------------------------- what a program has in hand

def _gen(seed, *more):
    g = torch.Generator(device="cuda")
    g.manual_seed(hash((int(seed),) + more) & 0x7FFFFFFF)
    return g


def _tables(N, Q, gaunt=True):
    T = c3d.quadrature(N, Q, with_m2=gaunt)
    if gaunt:
        _, T["row"], T["col"], T["val"] = c3d.gaunt_build(T["nm"], T["nm2"], T["nq"], T["M2"])
    return T


def _dev(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda")


def _edges(c):
    return c["nx"], c["ny"], c["nz"]


def _dt(c):
    n = _edges(c)
    if c["solver"] == "pn":
        return CFL * 0.5 * min(2.0 / e for e in n)
    return CFL * 2.0 / (2.0 + THETA) / sum(e / 2.0 for e in n)


def _axes(c, wrap):
    """Centres of the cells of the three axes with two ghosts on either side."""
    out = []
    for e in _edges(c):
        i = torch.arange(-2, e + 2, dtype=torch.float64, device="cuda")
        if wrap:
            i = i.remainder(e)
        out.append(-1.0 + (i + 0.5) * 2.0 / e)
    return torch.meshgrid(*out, indexing="ij")


def _sigma(c):
    """(sigma_t, sigma_s) of the cells."""
    s = torch.full([e + 4 for e in _edges(c)], c["sigma_s"], dtype=torch.float64, device="cuda")
    t = s.clone()
    if c["checker"]:
        b = c["checker"]
        i = [torch.arange(-2, e + 2, device="cuda").remainder(e) // b for e in _edges(c)]
        odd = (i[0][:, None, None] + i[1][None, :, None] + i[2][None, None, :]) % 2 == 1
        s[odd] = 10.0
        t = s + torch.where(odd, 0.1, 0.0)
    return t.reshape(-1).contiguous(), s.reshape(-1).contiguous()


def _moments(M, w, alpha):
    """<m e^{alpha.m}> of each row of alpha."""
    out = torch.empty_like(alpha)
    for a in range(0, len(alpha), 1 << 16):
        out[a:a + (1 << 16)] = (torch.exp(alpha[a:a + (1 << 16)] @ M.T) * w) @ M
    return out


def _fields(c, seed):
    """Moments and multipliers [cells, nm] of a problem's start, ghosts included."""
    nm = (c["N"] + 1) ** 2
    g = _gen(seed, 1)
    if c["field"] == "pulse":
        X = _axes(c, False)
        off = (torch.rand(3, dtype=torch.float64, device="cuda", generator=g) - 0.5) * 0.1
        s = c["width"] * (1.0 + 0.05 * float(torch.rand(1, device="cuda", generator=g)))
        r2 = sum((x - o) ** 2 for x, o in zip(X, off))
        G = torch.exp(-r2 / (2 * s * s)) / (s * math.sqrt(2 * math.pi)) ** 3
        u = torch.zeros(G.numel(), nm, dtype=torch.float64, device="cuda")
        u[:, 0] = 2.0 * math.sqrt(math.pi) * torch.clamp(G / (4 * math.pi), min=c["floor"]).reshape(-1)
        a = torch.zeros_like(u)
        a[:, 0] = math.sqrt(4 * math.pi) * torch.log(u[:, 0] / math.sqrt(4 * math.pi))
        return u, a
    # a transported field: smooth multipliers, anisotropy falling with the degree, and warm
    # starts that lag by what one time step changes
    X = _axes(c, True)
    l = torch.cat([torch.full((2 * n + 1,), float(n)) for n in range(c["N"] + 1)]).cuda()
    amp = (0.6 * 0.6 ** l).double()
    amp[0] = 2.0
    a = torch.zeros(X[0].numel(), nm, dtype=torch.float64, device="cuda")
    for k in range(1, 4):
        ph = torch.rand(3, nm, dtype=torch.float64, device="cuda", generator=g) * 2 * math.pi
        cf = torch.randn(nm, dtype=torch.float64, device="cuda", generator=g) * amp / k
        for m in range(nm):
            a[:, m] += (cf[m] * torch.cos(math.pi * k * X[0] + ph[0, m]) *
                        torch.cos(math.pi * X[1] + ph[1, m]) *
                        torch.cos(math.pi * X[2] + ph[2, m])).reshape(-1)
    T = c3d.quadrature(c["N"], c["Q"])
    u = _moments(_dev(T["M"]).reshape(T["nq"], nm), _dev(T["w"]), a)
    lag = 0.03 * torch.cos(math.pi * X[0]).reshape(-1, 1) + 0.02
    return u, a * (1.0 - lag)


class _Problem:
    """A resident problem with the moments and multipliers it starts from."""

    def __init__(self, c, seed, stream=None):
        self.c = c
        T = _tables(c["N"], c["Q"], c["solver"] == "mn" and c["hessian"] == "gaunt")
        kw = {}
        if c["solver"] == "pn":
            nm, nq = T["nm"], T["nq"]
            M = _dev(T["M"]).reshape(nq, nm)
            kw = dict(solver=0, pn_kinetic=int(c.get("flux") == "kinetic"),
                      pn_ops=_half_range(M, *(_dev(T[k]) for k in ("w", "xi", "eta", "mu")))
                      .cpu().numpy().reshape(-1))
        n = _edges(c)
        self.ctx = c3d.Context(nx=n[0], ny=n[1], nz=n[2], nm=T["nm"], nq=T["nq"], dx=2.0 / n[0],
                               dy=2.0 / n[1], dz=2.0 / n[2], M=T["M"], w=T["w"], xi=T["xi"],
                               eta=T["eta"], mu=T["mu"], theta=THETA, tol=TOL, ladder=LADDER,
                               stream=stream, **kw)
        if "row" in T:
            self.ctx.set_gaunt(T["nm2"], T["M2"], T["row"], T["col"], T["val"])
        if c["precision"] == "mixed":
            self.ctx.set_precision(1)
        self.u, self.a = _fields(c, seed)
        self.st, self.ss = _sigma(c)
        self.mn = c["solver"] == "mn"
        self.uo, self.ao = torch.empty_like(self.u), torch.empty_like(self.a)
        self.dt = _dt(c)
        torch.cuda.synchronize()

    def start(self):
        c3d.check(c3d.lib().c3d_set_state(self.ctx.h, self.u.data_ptr(),
                                          self.a.data_ptr() if self.mn else None,
                                          self.st.data_ptr(), self.ss.data_ptr(), 1), "set_state")

    def result(self):
        c3d.check(c3d.lib().c3d_get_state(self.ctx.h, self.uo.data_ptr(),
                                          self.ao.data_ptr() if self.mn else None, 1), "get_state")
        return [self.uo, self.ao] if self.mn else [self.uo]


class _Served:
    def __init__(self, c, seed):
        self.stream = torch.cuda.Stream()
        self.p = [_Problem(p, seed + 31 * i, ctypes.c_void_p(self.stream.cuda_stream))
                  for i, p in enumerate(_problems(c))]
        self.group = c3d.Group([p.ctx.h for p in self.p])

    def __del__(self):
        self.group.close()


class _Vectors:
    def __init__(self, c, seed):
        self.stream = torch.cuda.Stream()
        self.ctx, self.u0, self.a0, self.u, self.a = [], [], [], [], []
        for N in range(1, c["N"] + 1):
            T = _tables(N, 2 * (N + 3))
            ctx = c3d.Context(nx=2, ny=2, nz=2, nm=T["nm"], nq=T["nq"], dx=1.0, dy=1.0, dz=1.0,
                              M=T["M"], w=T["w"], xi=T["xi"], eta=T["eta"], mu=T["mu"],
                              batched=False, tol=TOL, ladder=LADDER,
                              stream=ctypes.c_void_p(self.stream.cuda_stream))
            ctx.set_gaunt(T["nm2"], T["M2"], T["row"], T["col"], T["val"])
            if c["precision"] == "mixed":
                ctx.set_precision(1)
            M, w = _dev(T["M"]).reshape(T["nq"], T["nm"]), _dev(T["w"])
            u = _moments(M, w, _seeded(c, seed, N, M, w))
            a = torch.zeros_like(u)
            a[:, 0] = 2 * math.sqrt(math.pi) * torch.log(u[:, 0] / (2 * math.sqrt(math.pi)))
            self.ctx.append(ctx)
            self.u0.append(u)
            self.a0.append(a)
            self.u.append(torch.empty_like(u))
            self.a.append(torch.empty_like(a))
        self.n = [c["n"]] * c["N"]
        self.group = c3d.Group([x.h for x in self.ctx])
        torch.cuda.synchronize()

    def __del__(self):
        self.group.close()


def _seeded(c, seed, N, M, w):
    """Multipliers of unit density whose higher components are N(0, s^2), s log-uniform."""
    g = _gen(seed, 2, N)
    n, nm = c["n"], (N + 1) ** 2
    s = torch.exp(torch.rand(n, 1, dtype=torch.float64, device="cuda", generator=g) *
                  math.log(c["smax"] / 0.1)) * 0.1
    a = torch.randn(n, nm, dtype=torch.float64, device="cuda", generator=g) * s
    a[:, 0] = 0.0
    a[:, 0] = -2.0 * math.sqrt(math.pi) * torch.log(_moments(M, w, a)[:, 0])
    return a


def _problems(c):
    """The problems of a serving pass: edges over [lo, hi], orders 1, 3, 5, early and late."""
    out = []
    for i in range(c["count"]):
        N = (1, 3, 5)[i % 3]
        e = c["lo"] + (c["hi"] - c["lo"]) * ((7 * i) % c["count"]) // max(1, c["count"] - 1)
        out.append(dict(kind="step", solver="mn", N=N, Q=2 * (N + 3), nx=e, ny=e, nz=e,
                        precision=c["precision"], hessian="gaunt", sigma_s=0.5 + 3.0 * i,
                        checker=0, field="aged" if i % 2 else "pulse", width=0.05 + 0.02 * i,
                        floor=1e-8, steps=1))
    return out


class _Host:
    """Host buffers of the reference's two offload calls."""


def _prepare_flux(c, seed):
    s = _Host()
    T = _tables(c["N"], c["Q"], False)
    field = dict(c, field="aged", solver="mn")
    s.alpha = _fields(field, seed)[1].cpu().numpy()
    s.flux = np.zeros_like(s.alpha)
    p = ctypes.POINTER(ctypes.c_double)
    s.keep = [T[k] for k in ("xi", "eta", "mu", "w", "M")]
    n = _edges(c)
    s.args = ([e + 4 for e in n] + [T["nm"], T["nq"]] + [2.0 / e for e in n] +
              [x.ctypes.data_as(p) for x in [s.alpha, s.flux] + s.keep] + [0])
    return s


def _prepare_hessian(c, seed):
    s = _Host()
    T = _tables(c["N"], c["Q"])
    nm, nm2, nq = T["nm"], T["nm2"], T["nq"]
    p, ip = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    M = _dev(T["M"]).reshape(nq, nm)
    s.alpha = _seeded(dict(c, smax=1.0), seed, c["N"], M, _dev(T["w"])).cpu().numpy()
    s.h = np.zeros((c["n"], nm, nm))
    g = int(c["form"] == "sparse")
    c3d.lib().solveHInit_cuda(nm, nm2, nq, c["n"], T["w"].ctypes.data_as(p),
                              T["M"].ctypes.data_as(p), T["M2"].ctypes.data_as(p), None,
                              T["val"].ctypes.data_as(p), T["col"].ctypes.data_as(ip),
                              T["row"].ctypes.data_as(ip), g)
    s.args = (nm, nm2, nq, c["n"], s.alpha.ctypes.data_as(p), s.h.ctypes.data_as(p), g, g)
    return s


def prepare(case, seed):
    make = dict(step=_Problem, serve=_Served, vectors=_Vectors, flux=_prepare_flux,
                hessian=_prepare_hessian)[case["kind"]]
    return case, make(case, seed)


def run(state):
    c, s = state
    if c["kind"] == "step":
        s.start()
        for _ in range(c["steps"]):
            s.ctx.step(s.dt)
        return s.result()
    if c["kind"] == "serve":
        for p in s.p:
            p.start()
        s.group.step([p.dt for p in s.p])
        return [p.result() for p in s.p]
    if c["kind"] == "vectors":
        with torch.cuda.stream(s.stream):
            for dst, src in zip(s.u + s.a, s.u0 + s.a0):
                dst.copy_(src)
        s.group.closure_vectors(s.n, [x.data_ptr() for x in s.u], [x.data_ptr() for x in s.a])
        return [s.u, s.a]
    if c["kind"] == "flux":
        c3d.lib().solveFluxKinetic_cuda(*s.args)
        return s.flux
    c3d.lib().solveH_cuda(*s.args)
    return s.h


# ---------------------------------------------------------------- what a pass cannot do without

def _step_work(c):
    nm, nq = (c["N"] + 1) ** 2, 2 * c["Q"] ** 2
    n = _edges(c)
    inner, cells = n[0] * n[1] * n[2], math.prod(e + 4 for e in n)
    stages = 2 * c["steps"]
    state = cells * (nm * 8.0 * (4 if c["solver"] == "mn" else 2) + 16.0)
    kinetic = inner * nq * (2.0 * nm + 60.0)
    if c["solver"] == "pn":
        flops = inner * 12.0 * nm * nm if c.get("flux") != "kinetic" else kinetic + cells * 2.0 * nm * nq
    else:
        # exponents, exponentials and moments of every cell once; three Hessians by the
        # extended moments and their Cholesky where every cell iterates
        flops = kinetic + cells * nq * (4.0 * nm + 1.0)
        if c["field"] == "aged":
            flops += 3.0 * cells * (nq * (2.0 * (2 * c["N"] + 1) ** 2 + 2.0 * nm) + nm ** 3 / 3.0)
    return state, stages * flops


def work(case):
    c = case
    if c["kind"] == "step":
        b, f = _step_work(c)
    elif c["kind"] == "serve":
        w = [_step_work(p) for p in _problems(c)]
        b, f = sum(x[0] for x in w), sum(x[1] for x in w)
    elif c["kind"] == "vectors":
        b = f = 0.0
        for N in range(1, c["N"] + 1):
            nm, nq = (N + 1) ** 2, 8 * (N + 3) ** 2
            b += c["n"] * nm * 32.0
            f += 5.0 * c["n"] * (nq * (2.0 * (2 * N + 1) ** 2 + 4.0 * nm) + nm ** 3 / 3.0)
    elif c["kind"] == "flux":
        nm, nq = (c["N"] + 1) ** 2, 2 * c["Q"] ** 2
        cells, inner = math.prod(e + 4 for e in _edges(c)), math.prod(_edges(c))
        b = cells * nm * 16.0
        f = cells * nq * (2.0 * nm + 1.0) + inner * nq * (2.0 * nm + 60.0)
    else:
        nm, nq = (c["N"] + 1) ** 2, 2 * c["Q"] ** 2
        b = c["n"] * (nm + nm * nm) * 8.0
        f = c["n"] * nq * (2.0 * nm + 2.0 * (2 * c["N"] + 1) ** 2)
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------- the same in plain torch

def _plain_tables(N, Q):
    """Basis [nq, nm] of orthonormal real spherical harmonics, weights and direction cosines."""
    x, wx = np.polynomial.legendre.leggauss(Q)
    ph = (np.arange(2 * Q) + 0.5) * np.pi / Q
    z, p = np.repeat(x, 2 * Q), np.tile(ph, Q)
    s = np.sqrt((1 - z) * (1 + z))
    P = {}
    for m in range(N + 1):
        v = np.full_like(z, math.sqrt((2 * m + 1) / (4 * np.pi)))
        for k in range(1, m + 1):
            v = v * -s * math.sqrt((2 * k - 1) / (2 * k))
        P[m, m] = v
        for l in range(m + 1, N + 1):
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1)) if l > m + 1 else 0.0
            P[l, m] = a * (z * P[l - 1, m] - (b * P[l - 2, m] if l > m + 1 else 0.0))
    r2 = math.sqrt(2.0)
    M = np.stack([P[l, 0] if m == 0 else r2 * P[l, abs(m)] * (np.cos(m * p) if m > 0 else np.sin(m * p))
                  for l in range(N + 1) for m in range(-l, l + 1)], axis=1)
    return [_dev(v) for v in (M, np.repeat(wx, 2 * Q) * np.pi / Q, s * np.cos(p), s * np.sin(p), z)]


def _half_range(M, w, xi, eta, mu):
    """The six half-range operators sum w c m m^T over c > 0, c <= 0 of each axis."""
    ops = []
    for c in (xi, eta, mu):
        for half in (c > 0, c <= 0):
            ops.append((M * (w * c * half)[:, None]).T @ M)
    return torch.stack(ops)


def _solve(M, w, u, a):
    """Multipliers whose moments are u, by Newton with halved steps from a."""
    scale = u[:, :1]
    m0 = float(M[0, 0])
    u, a = u / scale, a.clone()
    a[:, :1] -= torch.log(scale) / m0
    nq, nm = M.shape
    part = max(1, min(len(u), (1 << 27) // (nq * nm)))
    MM = None
    for lo in range(0, len(u), part):
        uu, aa = u[lo:lo + part], a[lo:lo + part].clone()
        todo = torch.arange(len(uu), device="cuda")
        for _ in range(60):
            e = torch.exp(aa[todo] @ M.T) * w
            g = e @ M - uu[todo]
            norm = g.norm(dim=1)
            keep = norm > 2e-14
            if not bool(keep.any()):
                break
            todo, e, g = todo[keep], e[keep], g[keep]
            H = torch.matmul((e[:, :, None] * M).transpose(1, 2), M)
            d = torch.cholesky_solve(-g[:, :, None], torch.linalg.cholesky_ex(H)[0])[:, :, 0]
            d = torch.nan_to_num(d)
            f = e.sum(1) - (aa[todo] * uu[todo]).sum(1)
            gd = (g * d).sum(1)
            t = torch.ones(len(todo), dtype=torch.float64, device="cuda")
            for _ in range(20):
                new = aa[todo] + t[:, None] * d
                fn = (torch.exp(new @ M.T) * w).sum(1) - (new * uu[todo]).sum(1)
                bad = ~(fn <= f + 1e-3 * t * gd + 1e-13 * f.abs())
                if not bool(bad.any()):
                    break
                t = torch.where(bad, 0.5 * t, t)
            aa[todo] += t[:, None] * d
            todo = todo[(t[:, None] * d).abs().amax(1) > 1e-14]
            if not len(todo):
                break
        a[lo:lo + part] = aa
    a[:, :1] += torch.log(scale) / m0
    return a


def _slope(l, c, r):
    def minmod(x, y):
        return torch.where(x * y > 0, torch.where(x.abs() < y.abs(), x, y), torch.zeros_like(x))
    return minmod(THETA * (r - c), minmod(0.5 * (r - l), THETA * (c - l)))


def _kinetic(c, values, M, w, cos):
    """sum_q m_q w_q Omega_q . (limited upwind differences of psi_q) on the interior cells;
    values(q0, q1): psi of some directions on the grid."""
    n = _edges(c)
    out = torch.zeros(math.prod(n), M.shape[1], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // math.prod(e + 4 for e in n))
    for q in range(0, len(w), step):
        psi = values(q, min(len(w), q + step))  # [nx+4, ny+4, nz+4, directions]
        total = 0.0
        for ax in range(3):
            h = 2.0 / n[ax]
            v = psi
            for other in range(3):
                if other != ax:
                    v = v.narrow(other, 2, n[other])
            at = [v.narrow(ax, k, n[ax]) for k in range(5)]
            up = (at[2] + 0.5 * _slope(at[1], at[2], at[3])) - (at[1] + 0.5 * _slope(at[0], at[1], at[2]))
            dn = (at[3] - 0.5 * _slope(at[2], at[3], at[4])) - (at[2] - 0.5 * _slope(at[1], at[2], at[3]))
            cq = cos[ax][q:q + step]
            total = total + torch.where(cq > 0, up, dn) * (cq * w[q:q + step] / h)
        out += total.reshape(-1, total.shape[-1]) @ M[q:q + step]
    return out


def _fill(c, u):
    """Periodic ghost faces (no edges, no corners) of u [nx+4, ny+4, nz+4, nm], in place."""
    n = _edges(c)
    for ax in range(3):
        v = u
        for other in range(3):
            if other != ax:
                v = v.narrow(other, 2, n[other])
        for k in (0, 1):
            v.select(ax, k).copy_(v.select(ax, n[ax] + k))
            v.select(ax, n[ax] + 2 + k).copy_(v.select(ax, 2 + k))


def _exact_step(c, seed):
    n, nm = _edges(c), (c["N"] + 1) ** 2
    M, w, *cos = _plain_tables(c["N"], c["Q"])
    u, a = _fields(c, seed)
    st, ss = (x.reshape([e + 4 for e in n])[2:-2, 2:-2, 2:-2].reshape(-1, 1) for x in _sigma(c))
    full = [e + 4 for e in n]
    grid = u.reshape(full + [nm])
    inner = grid[2:-2, 2:-2, 2:-2]
    dt = _dt(c)
    ops = _half_range(M, w, *cos) if c["solver"] == "pn" else None
    for _ in range(c["steps"]):
        old = inner.clone()
        for _ in range(2):
            _fill(c, grid)
            if c["solver"] == "pn" and c.get("flux") != "kinetic":
                flux = 0.0
                for ax in range(3):
                    v = grid
                    for other in range(3):
                        if other != ax:
                            v = v.narrow(other, 2, n[other])
                    b = [v.narrow(ax, k, n[ax]).reshape(-1, nm) for k in range(5)]
                    tp = 0.25 * b[3] + 0.75 * b[2] - 1.25 * b[1] + 0.25 * b[0]
                    tm = -0.25 * b[4] + 1.25 * b[3] - 0.75 * b[2] - 0.25 * b[1]
                    flux = flux + (tp @ ops[2 * ax].T + tm @ ops[2 * ax + 1].T) * (n[ax] / 2.0)
            elif c["solver"] == "pn":
                flux = _kinetic(c, lambda i, j: grid @ M[i:j].T, M, w, cos)
            else:
                a = _solve(M, w, u, a)
                flux = _kinetic(c, lambda i, j: torch.exp(a @ M[i:j].T).reshape(full + [-1]), M, w, cos)
            v = inner.reshape(-1, nm) * (1.0 - dt * st) - dt * flux
            v[:, :1] += dt * ss * inner.reshape(-1, nm)[:, :1]
            inner.copy_(v.reshape(inner.shape))
        inner.copy_(0.5 * (inner + old))
    return [u, a] if c["solver"] == "mn" else [u]


def exact(case, seed):
    """What run() returns, with every closure solved until its gradient is rounding error."""
    c = case
    # the plain form of the larger problems takes too long
    if c["kind"] == "step":
        nm, nq = (c["N"] + 1) ** 2, 2 * c["Q"] ** 2
        hess = 40.0 if c["field"] == "aged" else 8.0
        cost = math.prod(_edges(c)) * nq * c["steps"] * (hess * nm * nm if c["solver"] == "mn" else nm)
        return None if cost > 2e13 else _exact_step(c, seed)
    if c["kind"] == "serve":
        return [_exact_step(p, seed + 31 * i) for i, p in enumerate(_problems(c))]
    if c["kind"] == "vectors":
        a, u = [], []
        for N in range(1, c["N"] + 1):
            M, w = _plain_tables(N, 2 * (N + 3))[:2]
            a.append(_seeded(c, seed, N, M, w))
            u.append(_moments(M, w, a[-1]))
        return [u, a]
    M, w, *cos = _plain_tables(c["N"], c["Q"])
    if c["kind"] == "flux":
        full, nm = [e + 4 for e in _edges(c)], M.shape[1]
        a = _fields(dict(c, field="aged", solver="mn"), seed)[1]
        f = torch.zeros(full + [nm], dtype=torch.float64, device="cuda")
        inner = f[2:-2, 2:-2, 2:-2]
        k = _kinetic(c, lambda i, j: torch.exp(a @ M[i:j].T).reshape(full + [-1]), M, w, cos)
        inner.copy_(k.reshape(inner.shape))
        return f.reshape(-1, nm).cpu().numpy()
    a = _seeded(dict(c, smax=1.0), seed, c["N"], M, w)
    e = torch.exp(a @ M.T) * w
    h = torch.stack([(M * v[:, None]).T @ M for v in e])
    return h.cpu().numpy()
