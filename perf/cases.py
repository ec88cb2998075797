"""Performance cases of the framework's public entry points.

Each case is one pass of a user's program: time stepping of one solve in every
precision mode (`gpu.Solver`), a batched ensemble (`gpu.Ensemble`), the internal-force
call, and inference and training of the surrogate network (`nn.Network`).

    listed()          the named cases
    draw(rng)         one more case of the same ranges
    prepare(c, seed)  inputs made from the seed, and the handles a program keeps
    run(state)        one pass through the public entry points; returns its results
    work(c)           bytes and operations that the pass cannot do without
    exact(c, seed)    the same results in 64 bits by plain numpy and torch

Solves start from a superposition of plane waves of about six GLL points per wavelength
(the resolution meshes are sized for) or from rest, in a smooth random material, with a
moment source that is active during the pass; a pass advances a block of steps, fetches
the receiver rows and leaves the wavefield on the device.  The rows of the plain and
Kahan FP32 modes hold single-precision values and are kept as such.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from se2dr_fork_gb300 import gpu, host, nn, spec

ELEMENT = 31.25          # element edge in metres (the ensemble's)
VP, VP_VS, RHO = 5000.0, 1.73, 2700.0
COURANT = 0.3            # time step over (smallest node distance / fastest wave)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the reference demo's mesh in the reference's arithmetic, one logging block of the
        # application's loop (100 steps, norms, receiver rows): launch latency
        {"name": "fp64_demo8_p2", "kind": "step", "precision": "fp64", "mx": 8, "my": 8, "p": 2, "steps": 100, "nrec": 3, "nsrc": 2, "rest": True, "norms": True},
        # the 64 x 64, degree 6 validation solve in the reference's arithmetic
        {"name": "fp64_64_p6", "kind": "step", "precision": "fp64", "mx": 64, "my": 64, "p": 6, "steps": 40, "nrec": 1, "nsrc": 1, "rest": False, "norms": True},
        # a large reference-arithmetic solve of the heterogeneous workload's degree, ragged tiles
        {"name": "fp64_large_p4", "kind": "step", "precision": "fp64", "mx": 517, "my": 403, "p": 4, "steps": 4, "nrec": 64, "nsrc": 1, "rest": False, "norms": False},
        # two-float mode: the accurate FP32 solve
        {"name": "df_large_p4", "kind": "step", "precision": "fp32_df", "mx": 500, "my": 441, "p": 4, "steps": 6, "nrec": 64, "nsrc": 1, "rest": False, "norms": False},
        # one draw of the surrogate's training distribution solved alone
        {"name": "kahan_128_p4", "kind": "step", "precision": "fp32_kahan", "mx": 128, "my": 128, "p": 4, "steps": 100, "nrec": 16, "nsrc": 1, "rest": False, "norms": False},
        # the headline workload: the largest heterogeneous solve
        {"name": "kahan_2048_p4", "kind": "step", "precision": "fp32_kahan", "mx": 2048, "my": 2048, "p": 4, "steps": 10, "nrec": 64, "nsrc": 1, "rest": True, "norms": False},
        # degrees of the sweep that are not the headline's, odd sizes
        {"name": "kahan_large_p7", "kind": "step", "precision": "fp32_kahan", "mx": 333, "my": 301, "p": 7, "steps": 10, "nrec": 64, "nsrc": 1, "rest": False, "norms": False},
        {"name": "fp32_large_p2", "kind": "step", "precision": "fp32", "mx": 1001, "my": 873, "p": 2, "steps": 10, "nrec": 64, "nsrc": 1, "rest": False, "norms": False},
        # the internal force alone, as a host program's own time loop calls it on device vectors
        {"name": "force_fp64_p3", "kind": "force", "precision": "fp64", "mx": 163, "my": 158, "p": 3},
        # a batch of independent shots of uneven size and degree
        {"name": "ensemble_24", "kind": "ensemble", "shots": 24, "lo": 32, "hi": 256, "steps": 64, "block": 32, "nrec": 32},
        # surrogate serving and training at the repository's network configuration
        {"name": "surrogate_serve_64", "kind": "serve", "grid": 128, "width": 64, "modes": 16, "layers": 4, "batch": 64},
        {"name": "surrogate_train_32", "kind": "train", "grid": 128, "width": 64, "modes": 16, "layers": 4, "batch": 32, "steps": 8},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["force", "ensemble", "serve", "train"])
    if kind in ("step", "force"):
        precision = rng.choice(["fp64", "fp32_df", "fp32_kahan", "fp32_kahan", "fp32"])
        if kind == "force":
            precision = rng.choice(["fp64", "fp32"])
        p = rng.randint(1, 8)
        nodes = _log(rng, 300, {"fp64": 2.0e6, "fp32_df": 3.0e6}.get(precision, 1.6e7))
        ratio = rng.uniform(0.6, 1.6)
        mx = max(2, round(math.sqrt(nodes * ratio) / p))
        my = max(2, round(math.sqrt(nodes / ratio) / p))
        c = {"kind": kind, "precision": precision, "mx": mx, "my": my, "p": p}
        if kind == "step":
            most = {"fp64": 1.0e6, "fp32_df": 8.0e6}.get(precision, 1.0e8)
            c.update(steps=max(2, min(100, int(most / nodes))), nrec=rng.choice([1, 3, 16, 64]), nsrc=rng.randint(1, 2),
                     rest=rng.random() < 0.3, norms=rng.random() < 0.3)
        return c
    if kind == "ensemble":
        return {"kind": kind, "shots": rng.randint(2, 24), "lo": 32, "hi": rng.randint(64, 256), "steps": rng.randint(16, 64),
                "block": rng.choice([16, 32, 50]), "nrec": rng.choice([16, 32])}
    c = {"kind": kind, "grid": rng.choice([64, 96, 128]), "width": rng.choice([32, 48, 64]), "modes": rng.choice([8, 12, 16]),
         "layers": rng.randint(2, 4), "batch": max(1, round(_log(rng, 1, 64 if kind == "serve" else 32)))}
    if kind == "train":
        c["steps"] = rng.randint(2, 8)
    return c


def prepare(case, seed):
    return {"step": _prepare_step, "force": _prepare_force, "ensemble": _prepare_ensemble, "serve": _prepare_serve,
            "train": _prepare_train}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def exact(case, seed):
    return {"step": _exact_step, "force": _exact_force, "ensemble": _exact_ensemble, "serve": _exact_serve,
            "train": _exact_train}[case["kind"]](case, seed)


def work(case):
    kind = case["kind"]
    if kind == "step":
        b, f = _node_step(case["precision"], case["p"])
        n = _nodes(case) * case["steps"]
        return {"bytes": b * n, "flops": f * n}
    if kind == "force":
        size = 8 if case["precision"] == "fp64" else 4
        return {"bytes": (4 + 2 / case["p"] ** 2) * size * _nodes(case), "flops": _force_ops(case["p"]) * _nodes(case)}
    if kind == "ensemble":
        b = f = 0.0
        for s in _shot_sizes(case):
            n = (s[0] * s[2] + 1) * (s[1] * s[2] + 1) * case["steps"]
            bb, ff = _node_step("fp32_kahan", s[2])
            b, f = b + bb * n, f + ff * n
        return {"bytes": b, "flops": f}
    c = _net_config(case)
    pix, w, m, batch = c.ny * c.nx, c.width, c.modes, case["batch"]
    params = _net_params(c)
    dft = 2 * (c.ny * 2 * m * c.nx * w + 4 * m * 2 * c.ny * m * w)
    layer = 2 * dft + 2 * (2 * m * m) * 4 * w * w + 2 * pix * w * w
    dec = 2 * c.nrec * c.ny * c.hidden * (w + c.nout // c.ny)
    fwd = batch * (2 * pix * c.cin * w + c.layers * layer + dec)
    data = batch * (pix * 3 * 4 + c.nrec * c.nout * 4)
    if kind == "serve":
        return {"bytes": params * 4 + data, "flops": fwd}
    # per step: the batch's inputs and targets, p, m, v read and written
    return {"bytes": case["steps"] * (params * 4 * 6 + 2 * data), "flops": case["steps"] * (3 * fwd + 12 * params)}


def _nodes(c):
    return (c["mx"] * c["p"] + 1) * (c["my"] * c["p"] + 1)


def _force_ops(p):
    """Operations per node of the internal force: gradient and divergence along the row and
    the column of each GLL point, Hooke stress."""
    n1 = p + 1
    return (n1 * n1 / (p * p)) * (2 * (4 * 2 * n1) + 21)


def _node_step(precision, p):
    """(bytes, operations) of one node in one step."""
    if precision == "fp64":       # u, v, a read and written, M; lambda, mu per cell
        return 6 * 16 + 8 + 16 / p ** 2, _force_ops(p) + 16
    b = {"fp32": 32 + 4 + 8 / p ** 2, "fp32_kahan": 64 + 4 + 8 / p ** 2, "fp32_df": 64 + 8 + 16 / p ** 2}[precision]
    return b, {"fp32": 1, "fp32_kahan": 1, "fp32_df": 10}[precision] * _force_ops(p) + 20


# ---------------------------------------------------------------- solver inputs
def _gll(p):
    """GLL nodes and weights on [-1, 1] from the roots of P_p'."""
    c = np.zeros(p + 1)
    c[p] = 1.0
    leg = np.polynomial.legendre.Legendre(c)
    x = np.concatenate([[-1.0], np.sort(np.real(leg.deriv().roots())) if p > 1 else [], [1.0]])
    d1, d2 = leg.deriv(), leg.deriv(2)
    for _ in range(3):   # Newton on P_p'
        if p > 1:
            x[1:-1] -= d1(x[1:-1]) / d2(x[1:-1])
    return x, 2.0 / (p * (p + 1) * leg(x) ** 2)


def _derivative(x):
    """D[q, i] = derivative of Lagrange basis i at node q (barycentric form)."""
    n = len(x)
    diff = x[:, None] - x[None, :] + np.eye(n)
    w = 1.0 / np.prod(diff, axis=1)
    D = (w[None, :] / w[:, None]) / diff
    np.fill_diagonal(D, 0.0)
    np.fill_diagonal(D, -D.sum(axis=1))
    return D


def _axis(m, p, x, L):
    h = L / m
    e = (np.arange(m)[:, None] + 0.5 * (x[None, :p] + 1.0)).reshape(-1) * h
    return np.append(e, L)


def _random_field(mx, my, rng, corr=8.0):
    """Zero-mean, unit-variance smooth field on the cells [my, mx]."""
    ky, kx = np.fft.fftfreq(my)[:, None], np.fft.rfftfreq(mx)[None, :]
    f = np.fft.rfft2(rng.standard_normal((my, mx)).astype(np.float32)) * np.exp(-0.5 * (math.pi * corr) ** 2 * (kx ** 2 + ky ** 2))
    v = np.fft.irfft2(f, s=(my, mx)).astype(np.float64)
    return (v - v.mean()) / max(v.std(), 1e-12)


class _Problem:
    """The inputs of one solve, made from the seed alone."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        self.mx, self.my, self.p = case["mx"], case["my"], case["p"]
        self.Lx, self.Ly = self.mx * ELEMENT, self.my * ELEMENT
        vp = VP * (1.0 + 0.1 * np.clip(_random_field(self.mx, self.my, rng), -3, 3))
        self.vp, self.vs, self.rho = vp, vp / VP_VS, np.full_like(vp, RHO)
        self._finish(rng, case)

    def _finish(self, rng, case):
        x, _ = _gll(self.p)
        self.steps = case.get("steps", 0)
        self.dt = float(COURANT * 0.5 * ELEMENT * (x[1] - x[0]) / self.vp.max())
        inner = lambda L: float(rng.uniform(0.25 * L, 0.75 * L))  # noqa: E731
        self.sources = []
        for _ in range(case.get("nsrc", 0)):
            m = rng.standard_normal(3) * 1e15
            self.sources.append((inner(self.Lx), inner(self.Ly), (m[0], m[1], m[1], m[2]),
                                 (float(rng.uniform(0.2, 0.8)) * max(self.steps, 1) * self.dt, float(rng.uniform(5, 20)), 1.0)))
        n = case.get("nrec", 0)
        y = float(rng.uniform(0.3, 0.7)) * self.Ly
        self.receivers = [(float(v), y) for v in np.linspace(0.1 * self.Lx, 0.9 * self.Lx, n) + rng.uniform(-3, 3, n)]
        # plane waves: (amplitudes, wave vector, phase)
        self.waves = []
        for _ in range(6):
            a, k = rng.uniform(0, 2 * math.pi), 2 * math.pi / (6.0 / self.p * ELEMENT) * rng.uniform(0.5, 1.0)
            self.waves.append((rng.standard_normal(2) * 1e-4, (k * math.cos(a), k * math.sin(a)), rng.uniform(0, 2 * math.pi)))
        self.rest = bool(case.get("rest", False))

    def setup(self):
        sp = spec.Spec(mx=self.mx, my=self.my, p=self.p, scale=(self.Lx, self.Ly), shift=(0.0, 0.0), vp=VP, vs=VP / VP_VS,
                       rho=RHO, cell_vp=self.vp, cell_vs=self.vs, cell_rho=self.rho, dt=self.dt, tmax=1.0e30, nt=1000,
                       nearest_internal_gll=self.p > 1, receivers=self.receivers,
                       sources=[spec.Source(s[0], s[1], s[2], spec.STF_RICKER, s[3]) for s in self.sources])
        return host.Setup(sp)

    def fields(self):
        """u, v, a [ny, nx, 2] of the initial state."""
        xi, _ = _gll(self.p)
        x, y = _axis(self.mx, self.p, xi, self.Lx), _axis(self.my, self.p, xi, self.Ly)
        out = np.zeros((3, len(y), len(x), 2))
        if not self.rest:
            for amp, k, ph in self.waves:
                om = VP * math.hypot(*k)
                cx, sx, cy, sy = np.cos(k[0] * x), np.sin(k[0] * x), np.cos(k[1] * y + ph), np.sin(k[1] * y + ph)
                re, im = np.outer(cy, cx) - np.outer(sy, sx), np.outer(sy, cx) + np.outer(cy, sx)
                for c in range(2):
                    out[0, :, :, c] += amp[c] * re
                    out[1, :, :, c] += amp[c] * om * im
                    out[2, :, :, c] -= amp[c] * om * om * re
        return out


class _Device:
    """A device array of a solver as an object that torch can view; it keeps the solver."""

    def __init__(self, solver, ptr, shape, strides, typestr):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides, "typestr": typestr, "version": 3}


def _device_fields(st):
    """The solver's u, v, a on the device, [ny, nx, 2] without the row padding."""
    i, out = st["info"], []
    size, kind = (8, "<f8") if i["precision"] == gpu.FP64 else (4, "<f4")
    for ptr in st["solver"].device_fields():
        if ptr not in st["views"]:
            st["views"][ptr] = torch.as_tensor(_Device(st["solver"], ptr, (i["ny_g"], i["nx_g"], 2), (i["pitch"] * 2 * size, 2 * size, size), kind), device="cuda")
        out.append(st["views"][ptr])
    return out


def _prepare_step(case, seed):
    pb = _Problem(case, seed)
    s = gpu.Solver(pb.setup(), case["precision"], trace_capacity=case["steps"])
    if not pb.rest:
        s.set_fields(*[f.reshape(-1) for f in pb.fields()])
    return {"run": _run_step, "solver": s, "steps": case["steps"], "norms": case["norms"], "info": s.info(), "views": {},
            "rows": np.float32 if case["precision"] in ("fp32", "fp32_kahan") else np.float64}


def _run_step(st):
    s = st["solver"]
    s.advance(st["steps"])
    out = {"norms": s.norms()} if st["norms"] else {}
    out["rows"] = s.traces().astype(st["rows"], copy=False)
    out["u"], out["v"], out["a"] = _device_fields(st)
    return out


def _prepare_force(case, seed):
    pb = _Problem(case, seed)
    s = gpu.Solver(pb.setup(), case["precision"])
    u = torch.as_tensor(pb.fields()[0].reshape(-1), dtype=torch.float64 if case["precision"] == "fp64" else torch.float32).cuda()
    return {"run": _run_force, "solver": s, "u": u, "F": torch.zeros_like(u)}


def _run_force(st):
    st["solver"].assemble_linear_form_device(st["u"].data_ptr(), st["F"].data_ptr())
    return st["F"]


# ---------------------------------------------------------------- 64-bit solve
class _Solve64:
    """The solve by dense element contractions in float64 torch."""

    def __init__(self, pb):
        dev = "cuda"
        self.pb, p = pb, pb.p
        xi, w = _gll(p)
        self.n1, self.nx, self.ny = p + 1, pb.mx * p + 1, pb.my * p + 1
        self.D = torch.as_tensor(_derivative(xi), device=dev)
        self.x, self.y = _axis(pb.mx, p, xi, pb.Lx), _axis(pb.my, p, xi, pb.Ly)
        self.jac = ELEMENT / 2
        self.W = torch.as_tensor(np.outer(w, w) * self.jac ** 2, device=dev)           # [b, a]
        mu = torch.as_tensor(pb.rho * pb.vs ** 2, device=dev)[:, :, None, None]
        lam = torch.as_tensor(pb.rho * pb.vp ** 2, device=dev)[:, :, None, None] - 2 * mu
        self.lam, self.mu = lam, mu
        rho = torch.as_tensor(pb.rho, device=dev)
        M = torch.zeros(self.ny, self.nx, dtype=torch.float64, device=dev)
        for b in range(self.n1):
            for a in range(self.n1):
                M[b:b + (pb.my - 1) * p + 1:p, a:a + (pb.mx - 1) * p + 1:p] += rho * self.W[b, a]
        self.M = M[:, :, None]
        self.sources = [self._source(s) for s in pb.sources]
        self.recs = [self._nearest(r, 0) for r in pb.receivers]

    def _nearest(self, xy, lo):
        """Element (ex, ey) of a point and its nearest GLL point (a, b), without the `lo` outer ones."""
        p = self.pb.p
        ex, ey = min(int(xy[0] / ELEMENT), self.pb.mx - 1), min(int(xy[1] / ELEMENT), self.pb.my - 1)
        a = lo + int(np.argmin(np.abs(self.x[ex * p + lo:ex * p + p + 1 - lo] - xy[0])))
        b = lo + int(np.argmin(np.abs(self.y[ey * p + lo:ey * p + p + 1 - lo] - xy[1])))
        return ex, ey, a, b

    def _source(self, s):
        """(node window, values [b, a, 2], wavelet) of a moment source: M : grad N at its GLL point."""
        p = self.pb.p
        ex, ey, a, b = self._nearest(s[:2], 1 if p > 1 else 0)
        gx, gy = torch.zeros(self.n1, self.n1, dtype=torch.float64), torch.zeros(self.n1, self.n1, dtype=torch.float64)
        D = self.D.cpu()
        gx[b, :] = D[a] / self.jac
        gy[:, a] = D[b] / self.jac
        m = s[2]
        g = torch.stack([m[0] * gx + m[1] * gy, m[2] * gx + m[3] * gy], dim=2).cuda()
        return (slice(ey * p, ey * p + p + 1), slice(ex * p, ex * p + p + 1)), g, s[3]

    def _grad(self, f):
        """d/dx, d/dy [ey, ex, b, a] of a nodal scalar [ny, nx] at every element's GLL points."""
        p, n1, sy = self.pb.p, self.n1, f.stride(0)
        e = f.as_strided((self.pb.my, self.pb.mx, n1, n1), (p * sy, p * f.stride(1), sy, f.stride(1)), f.storage_offset())
        return torch.matmul(e, self.D.T) / self.jac, torch.matmul(self.D, e) / self.jac

    def force(self, u):
        """-(sum over elements of B^T sigma) for u [ny, nx, 2]."""
        p = self.pb.p
        exx, uxy = self._grad(u[:, :, 0])
        uyx, eyy = self._grad(u[:, :, 1])
        sxy = self.mu * (uxy + uyx) * self.W
        sxx = ((self.lam + 2 * self.mu) * exx + self.lam * eyy) * self.W
        syy = (self.lam * exx + (self.lam + 2 * self.mu) * eyy) * self.W
        F = torch.zeros_like(u)
        for c, (sx, sy) in enumerate(((sxx, sxy), (sxy, syy))):
            fe = -(torch.matmul(sx, self.D) + torch.matmul(self.D.T, sy)) / self.jac
            for b in range(self.n1):
                for a in range(self.n1):
                    F[b:b + (self.pb.my - 1) * p + 1:p, a:a + (self.pb.mx - 1) * p + 1:p, c] += fe[:, :, b, a]
        return F

    def advance(self, n, state=None):
        """Newmark (beta 0, gamma 1/2) steps; returns (u, v, a, receiver rows)."""
        dt = self.pb.dt
        u, v, a = [torch.as_tensor(f).cuda() for f in self.pb.fields()] if state is None else state
        t, rows = 0.0, []
        for _ in range(n):
            t += dt
            u = u + dt * v + 0.5 * dt * dt * a
            v = v + 0.5 * dt * a
            F = self.force(u)
            for win, g, (t0, f0, amp) in self.sources:
                q = (math.pi * f0 * (t - t0)) ** 2
                F[win] += amp * (1 - 2 * q) * math.exp(-q) * g
            a = F / self.M
            v = v + 0.5 * dt * a
            rows.append(self._row(t, u, v, a))
        return u, v, a, (torch.stack(rows).cpu().numpy() if rows else None)

    def _row(self, t, u, v, a):
        p, out = self.pb.p, []
        for ex, ey, ia, ib in self.recs:
            Y, X = ey * p + ib, ex * p + ia
            curl = (self.D[ia] @ v[Y, ex * p:ex * p + p + 1, 1] - self.D[ib] @ v[ey * p:ey * p + p + 1, X, 0]) / self.jac
            out += [u[Y, X], v[Y, X], a[Y, X], curl.reshape(1)]
        return torch.cat([torch.tensor([t], dtype=torch.float64, device="cuda")] + out)


def _exact_step(case, seed):
    pb = _Problem(case, seed)
    u, v, a, rows = _Solve64(pb).advance(case["steps"])
    out = {}
    if case["norms"]:
        out["norms"] = np.array([float(x) for f in (u, v) for x in (f.max(), f.min(), f.norm())])
    out["rows"] = rows
    if case["precision"] != "fp64":   # the FP32 modes hold the leapfrog state: v + dt/2 a, and u of the next step
        v = v + 0.5 * pb.dt * a
        u = u + pb.dt * v
    out["u"], out["v"], out["a"] = u, v, a
    return out


def _exact_force(case, seed):
    pb = _Problem(case, seed)
    return _Solve64(pb).force(torch.as_tensor(pb.fields()[0]).cuda()).reshape(-1)


# ---------------------------------------------------------------- ensemble
def _shot_sizes(case):
    """Mesh and degree of every shot: the case alone decides them, so that a case is the same work for every seed."""
    rng = np.random.default_rng([case["shots"], case["lo"], case["hi"], case["steps"]])
    return [(int(rng.integers(case["lo"], case["hi"] + 1)), int(rng.integers(case["lo"], case["hi"] + 1)), int(rng.choice([3, 4, 6])))
            for _ in range(case["shots"])]


class _Shot(_Problem):
    """Two layers and an elliptical inclusion, receivers along the surface, start at rest."""

    def __init__(self, case, size, rng):
        self.mx, self.my, self.p = size
        self.Lx, self.Ly = self.mx * ELEMENT, self.my * ELEMENT
        x, y = (np.arange(self.mx) + 0.5) / self.mx, (np.arange(self.my) + 0.5) / self.my
        r = rng.uniform(0.1, 0.3, 2)
        inside = ((x[None, :] - rng.uniform(0.3, 0.7)) / r[0]) ** 2 + ((y[:, None] - rng.uniform(0.2, 0.6)) / r[1]) ** 2 < 1
        where = np.where(inside, 2, (y[:, None] < rng.uniform(0.4, 0.8)).astype(int) + np.zeros((1, self.mx), dtype=int))
        vp = rng.uniform(3000, 6000, 3)
        self.vp, self.vs, self.rho = vp[where], (vp / rng.uniform(1.6, 1.9, 3))[where], rng.uniform(2000, 3000, 3)[where]
        self._finish(rng, dict(case, nsrc=1, rest=True))
        self.receivers = [(xr, self.Ly - 1e-3) for xr, _ in self.receivers]


def _shots(case, seed):
    rng = np.random.default_rng(seed)
    return [_Shot(case, size, rng) for size in _shot_sizes(case)]


def _prepare_ensemble(case, seed):
    e = gpu.Ensemble([s.setup() for s in _shots(case, seed)], "fp32_kahan", block=case["block"])
    return {"run": _run_ensemble, "ensemble": e, "steps": case["steps"]}


def _run_ensemble(st):
    return np.concatenate(st["ensemble"].advance(st["steps"]), axis=1).astype(np.float32)


def _exact_ensemble(case, seed):
    return np.concatenate([_Solve64(s).advance(case["steps"])[3] for s in _shots(case, seed)], axis=1)


# ---------------------------------------------------------------- surrogate
def _net_config(case):
    g = case["grid"]
    return nn.Config(ny=g, nx=g, cin=16, width=case["width"], modes=case["modes"], layers=case["layers"], nrec=16, nout=16 * g,
                     hidden=128, max_batch=case["batch"])


def _net_shapes(c):
    w, m, ns = c.width, c.modes, c.nout // c.ny
    shapes = [("W0", (c.cin, w), c.cin), ("b0", (w,), 0)]
    for i in range(c.layers):
        shapes += [("R%d" % i, (2 * m, m, w, w), w * w), ("I%d" % i, (2 * m, m, w, w), w * w), ("W%d" % (i + 1), (w, w), w), ("b%d" % (i + 1), (w,), 0)]
    return shapes + [("V1", (w, c.hidden), w), ("c1", (c.hidden,), 0), ("V2", (c.hidden, ns), c.hidden), ("c2", (ns,), 0)]


def _net_params(c):
    return sum(math.prod(s) for _, s, _ in _net_shapes(c))


class _NetData:
    """Parameters, and a resident data set of draws: materials, source cells, targets."""

    def __init__(self, case, seed, samples):
        self.c = c = _net_config(case)
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        uni = lambda *s: 2 * torch.rand(*s, generator=g, device="cuda") - 1  # noqa: E731
        self.params = torch.cat([(uni(math.prod(s)) / math.sqrt(fan) if fan else 0.05 * uni(math.prod(s))) for _, s, fan in _net_shapes(c)])
        self.rec = [(2 * r + 1) * c.nx // (2 * c.nrec) for r in range(c.nrec)]
        y, x = torch.arange(c.ny, device="cuda")[None, :, None], torch.arange(c.nx, device="cuda")[None, None, :]
        box = uni(samples, 4, 1, 1)
        top = (y < c.ny * (0.6 + 0.2 * box[:, 0])).float()
        hole = (((x / c.nx - 0.5 - 0.2 * box[:, 1]) / 0.2) ** 2 + ((y / c.ny - 0.4 - 0.2 * box[:, 2]) / 0.15) ** 2 < 1).float()
        layers = torch.tensor([4500.0, 2600.0, 2500.0], device="cuda") * (1 + 0.3 * uni(samples, 3, 3))
        self.mat = torch.where(hole[..., None] > 0, layers[:, None, None, 2], torch.where(top[..., None] > 0, layers[:, None, None, 0], layers[:, None, None, 1])).contiguous()
        self.src = (torch.rand(samples, 2, generator=g, device="cuda") * torch.tensor([0.8 * c.nx, 0.4 * c.ny], device="cuda") + 4).contiguous()
        t = torch.linspace(0, 1, c.nout, device="cuda")
        f = 4 + 3 * uni(samples, c.nrec, 1)
        self.target = (torch.sin(2 * math.pi * f * (t - 0.2 * uni(samples, c.nrec, 1))) * torch.exp(-((t - 0.5) / 0.3) ** 2)).contiguous()
        self.order = torch.randperm(samples, generator=g, device="cuda").to(torch.int32)

    def network(self):
        n = nn.Network(self.c, seed=0)
        n.set_params(self.params.cpu().numpy())
        n.set_receivers(self.rec)
        return n


SIGMA = 2.0


def _prepare_serve(case, seed):
    d = _NetData(case, seed, case["batch"])
    c = d.c
    x = torch.zeros(case["batch"], c.ny, c.nx, c.cin, dtype=torch.bfloat16, device="cuda")
    return {"run": _run_serve, "net": d.network(), "data": d, "x": x, "out": torch.zeros(case["batch"], c.nrec, c.nout, device="cuda")}


def _run_serve(st):
    d = st["data"]
    st["net"].build_inputs(d.mat, d.src, d.order, SIGMA, st["x"])
    st["net"].forward(st["x"], st["out"])
    return st["out"]


def _prepare_train(case, seed):
    d = _NetData(case, seed, case["batch"] * case["steps"])
    c, b = d.c, case["batch"]
    return {"run": _run_train, "net": d.network(), "data": d, "batches": list(d.order.view(-1, b).unbind(0)),
            "x": torch.zeros(b, c.ny, c.nx, c.cin, dtype=torch.bfloat16, device="cuda"),
            "t": torch.zeros(b, c.nrec, c.nout, device="cuda")}


LR = 1e-3


def _run_train(st):
    """A run of optimizer steps over the data set, then the weights."""
    net, d, losses = st["net"], st["data"], []
    for idx in st["batches"]:
        net.build_inputs(d.mat, d.src, idx, SIGMA, st["x"])
        net.gather_targets(d.target, idx, st["t"])
        losses.append(net.loss_grad(st["x"], st["t"]))
        net.adam_step(LR)
    return {"losses": losses, "params": net.params()}


def _inputs64(d, idx):
    """The network's input channels [b, row from the top, x, 6] of the draws idx."""
    c, idx = d.c, idx.long()
    mat = d.mat[idx].double().flip(1)
    src = d.src[idx].double()
    x, y = torch.arange(c.nx, device="cuda").double(), torch.arange(c.ny, device="cuda").double()
    mat = (mat - torch.tensor([5000.0, 2800.0, 2500.0], device="cuda").double()) / torch.tensor([1500.0, 800.0, 500.0], device="cuda").double()
    r2 = (x + 0.5 - src[:, 0, None, None]) ** 2 + (y[:, None] + 0.5 - (c.ny - src[:, 1, None, None])) ** 2
    one = torch.ones_like(r2)
    return torch.cat([mat, torch.exp(-r2 / (2 * SIGMA ** 2))[..., None], (one * ((2 * x + 1) / c.nx - 1))[..., None],
                      (one * ((2 * y + 1) / c.ny - 1)[:, None])[..., None]], dim=3)


def _forward64(d, P, x):
    c, m = d.c, d.c.modes
    ky = torch.tensor([j if j < m else j - 2 * m for j in range(2 * m)], device="cuda").double()
    grid = lambda n, k: torch.polar(torch.ones(len(k), n, device="cuda").double(), -2 * math.pi * k[:, None] * torch.arange(n, device="cuda").double() / n)  # noqa: E731
    Ey, Ex = grid(c.ny, ky), grid(c.nx, torch.arange(m, device="cuda").double())
    scale = (torch.where(torch.arange(m, device="cuda") == 0, 1.0, 2.0).double() / (c.nx * c.ny))[:, None]
    h = x @ P["W0"][:x.shape[3]] + P["b0"]
    for i in range(c.layers):
        z = torch.einsum("jy,byqc->bjqc", Ey, torch.einsum("qx,byxc->byqc", Ex, h.to(Ey.dtype)))
        z = torch.einsum("bjqc,jqcd->bjqd", z, torch.complex(P["R%d" % i], P["I%d" % i]))
        s = torch.einsum("qx,byqc->byxc", Ex.conj() * scale, torch.einsum("jy,bjqc->byqc", Ey.conj(), z)).real
        h = s + h @ P["W%d" % (i + 1)] + P["b%d" % (i + 1)]
        if i < c.layers - 1:
            h = torch.nn.functional.gelu(h)
    h = h[:, :, d.rec].permute(0, 2, 1, 3)
    h = torch.nn.functional.gelu(h @ P["V1"] + P["c1"]) @ P["V2"] + P["c2"]
    return h.reshape(x.shape[0], c.nrec, c.nout)


def _unpack64(d, flat):
    out, o = {}, 0
    for name, s, _ in _net_shapes(d.c):
        out[name] = flat[o:o + math.prod(s)].view(s)
        o += math.prod(s)
    return out


def _exact_serve(case, seed):
    d = _NetData(case, seed, case["batch"])
    P = _unpack64(d, d.params.double())
    with torch.no_grad():
        return torch.cat([_forward64(d, P, _inputs64(d, i)) for i in d.order.split(16)])


def _exact_train(case, seed):
    d = _NetData(case, seed, case["batch"] * case["steps"])
    p = d.params.double().requires_grad_()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for k, idx in enumerate(d.order.view(-1, case["batch"]).unbind(0)):
        total, grad = 0.0, torch.zeros_like(m)
        for part in idx.split(8):
            out = _forward64(d, _unpack64(d, p), _inputs64(d, part))
            loss = ((out - d.target[part.long()].double()) ** 2).sum() / (len(idx) * d.c.nrec * d.c.nout)
            grad += torch.autograd.grad(loss, p)[0]
            total += float(loss)
        losses.append(total)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad ** 2
            p -= LR * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"losses": losses, "params": p.detach()}
