"""The measured workloads of this framework, each through its public Python API.

A case is a dict of plain values: the path (which entry point a program calls),
the mesh (n nodes per axis and element, mx x my x mz elements of the unit cube,
warp amplitude), the state's type, Kreiss-Oliger dissipation, the outer boundary
and how many steps one call makes.  The paths:

  rk4    step_rk4_curved on an ADM background: the call inside every solve loop
  tsit5  step_erk_curved: the integrator the solver picks for n = 5 and 6
  rhs    wave3d_curved_rhs: one evaluation, for programs with their own integrator
  host   evolve_curved_host: samples and energies copied to host buffers, as evolve3d does
  sipg   step_rk4_sipg: the second-order (SIPG) system on a flat cube
  strong wave_strong_rhs_mesh: the strong-form second-order right-hand side
  batch  Batch.step: many small solves of mixed order advanced together

exact() evaluates the same discretisations with plain torch in 64 bits: the
operators, the geometry and the backgrounds are written here from their
formulas, nothing comes from the package.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wavetoysecondorder.jl_b200")
_CTX = []


def _wt():
    if "wavetoy_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("wavetoy_b200", os.path.join(_PKG, "__init__.py"),
                                                      submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["wavetoy_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["wavetoy_b200"]


def _ctx():
    if not _CTX:
        _CTX.append(_wt().Context(0))
    return _CTX[0]


def _case(name, path, n, m, **more):
    c = {"path": path, "n": n, "mx": m[0], "my": m[1], "mz": m[2], "warp": 0.05, "dtype": "f64", "eps_ko": 0.0,
         "bc": "sommerfeld", "steps": 1, "samples": 1, "metric": True}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the flat standing wave of the test-suite, 4^3 elements, n = 6, with dissipation: the smallest solve
        _case("sipg_n6_4cubed", "sipg", 6, (4, 4, 4), warp=0.0, eps_ko=0.1, steps=10),
        # the same system at production size
        _case("sipg_n6_40cubed", "sipg", 6, (40, 40, 40), warp=0.0, eps_ko=0.1),
        # the solver's defaults (n = 4, 8 elements per axis): the steps between two samples of a small run
        _case("rk4_n4_8cubed", "rk4", 4, (8, 8, 8), warp=0.0, steps=10),
        # warped ADM pulse, 16^3 elements, n = 8: an ordinary run
        _case("rk4_n8_16cubed", "rk4", 8, (16, 16, 16), steps=4),
        # the large warped ADM solve in both state types (FP32: the compensated default form)
        _case("rk4_n8_40cubed", "rk4", 8, (40, 40, 40)),
        _case("rk4_n8_40cubed_f32", "rk4", 8, (40, 40, 40), dtype="f32"),
        # a dissipative run (the right-hand side's default eps_KO)
        _case("rk4_ko_n8_24cubed", "rk4", 8, (24, 24, 24), eps_ko=0.1),
        # the integrator chosen for n = 5, 6
        _case("tsit5_n6_24cubed", "tsit5", 6, (24, 24, 24), steps=2),
        # one evaluation on an uneven mesh of an order without special kernels, with the default dissipation
        _case("rhs_ko_n7_ragged", "rhs", 7, (17, 13, 11), eps_ko=0.1, bc="full_dirichlet"),
        # samples and energies to the host while it runs
        _case("host_n8_16cubed", "host", 8, (16, 16, 16), steps=2, samples=4),
        # the strong form on a warped cube
        _case("strong_n5_28cubed", "strong", 5, (28, 28, 28)),
        # a served mix of small solves, n = 4, 6, 8
        _case("batch_f32_24", "batch", 0, (4, 4, 10), dtype="f32", steps=2, count=24, mix=7),
    ]


def draw(rng):
    path = rng.choice(["rk4", "rk4", "rk4", "tsit5", "rhs", "host", "sipg", "strong", "batch"])
    if path == "batch":
        lo = rng.randint(3, 5)
        return _case(None, "batch", 0, (lo, lo, rng.randint(lo + 2, 11)), dtype=rng.choice(["f32", "f32", "f64"]),
                     steps=rng.randint(1, 4), count=rng.randint(6, 28), mix=rng.randrange(1 << 20))
    n = rng.choice({"rk4": [4, 5, 6, 7, 8, 8, 8], "tsit5": [5, 6], "rhs": [4, 5, 6, 7, 8], "host": [4, 6, 8],
                    "sipg": [4, 5, 6, 7, 8], "strong": [4, 5, 6, 7, 8]}[path])
    ko = path in ("rk4", "rhs", "sipg") and rng.random() < 0.4
    top = {"rk4": 12e6, "tsit5": 3e6, "rhs": 6e6, "host": 3e6, "sipg": 8e6, "strong": 6e6}[path] * (0.5 if ko else 1)
    nodes = math.exp(rng.uniform(math.log(64 * n ** 3), math.log(top)))
    e = (nodes / n ** 3) ** (1 / 3)
    m = [max(2, round(e * rng.uniform(0.75, 1.3))) for _ in range(3)]
    if ko:  # mu is the spectral radius along x: the finest axis first
        m.sort(reverse=True)
    return _case(None, path, n, m, warp=0.0 if path == "sipg" else rng.choice([0.0, 0.03, 0.05]),
                 dtype=rng.choice(["f64", "f64", "f32"]), eps_ko=0.1 if ko else 0.0,
                 bc=rng.choice(["sommerfeld", "sommerfeld", "full_dirichlet"]) if path in ("rk4", "rhs") else
                 "sommerfeld",
                 steps=rng.randint(1, 6 if nodes < 2e6 else 2) if path not in ("rhs", "strong") else 1,
                 samples=rng.randint(2, 5) if path == "host" else 1,
                 metric=True)


# ---- inputs (from the seed alone) ----------------------------------------------------


def _members(case):
    """The (n, elements per axis) of a batch's solves."""
    r = random.Random(case["mix"])
    return [((4, 6, 8)[k % 3], r.randint(case["mx"], case["mz"])) for k in range(case["count"])]


def _gll(n):
    """GLL nodes and weights on [0, 1] and the differentiation matrix."""
    leg = np.polynomial.legendre.Legendre.basis(n - 1)
    d1, d2 = leg.deriv(), leg.deriv(2)
    x = np.sort(np.concatenate([[-1.0], d1.roots().real, [1.0]]))
    for _ in range(3):
        x[1:-1] -= d1(x[1:-1]) / d2(x[1:-1])
    x = 0.5 * (x - x[::-1])
    p = leg(x)
    w = 2.0 / (n * (n - 1) * p * p)
    d = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                d[i, j] = p[i] / (p[j] * (x[i] - x[j]))
    d -= np.diag(d.sum(axis=1))
    return 0.5 * (x + 1.0), 0.5 * w, 2.0 * d


def _axes(case, dev):
    """The reference coordinates s in [0, 1] of the nodes, shaped [ez, ey, ex, k, j, i]."""
    n, m = case["n"], (case["mx"], case["my"], case["mz"])
    x = torch.tensor(_gll(n)[0], dtype=torch.float64, device=dev)
    s = [(torch.arange(m[a], dtype=torch.float64, device=dev)[:, None] + x) / m[a] for a in range(3)]
    full = (m[2], m[1], m[0], n, n, n)
    return [s[0].view(1, 1, m[0], 1, 1, n).expand(full), s[1].view(1, m[1], 1, 1, n, 1).expand(full),
            s[2].view(m[2], 1, 1, n, 1, 1).expand(full)]


def _coords(case, dev):
    s = _axes(case, dev)
    if not case["warp"]:
        return s
    p = case["warp"] * torch.sin(2 * math.pi * s[0]) * torch.sin(2 * math.pi * s[1]) * torch.sin(2 * math.pi * s[2])
    return [a + p for a in s]


def _adm(seed):
    """alpha = 1 + p0 sin 2 pi x, beta = p1 cos 2 pi x_i, gamma = 1 + p2 exp(-r^2/p3)(1 + s/2)."""
    r = random.Random(seed)
    return [0.05, 0.02, 0.1, 0.05, 0.5, 0.5, 0.5] + [r.uniform(-0.2, 0.2) for _ in range(6)]


def _fields(case, seed, dev):
    """Two pulses in each of the two fields; sipg: a standing wave of seeded amplitude plus pulses."""
    r = random.Random(seed + 1)
    x = _coords(case, dev)
    out = []
    for f in range(2):
        u = torch.zeros_like(x[0], memory_format=torch.contiguous_format)
        for _ in range(2):
            c, a, w = [r.uniform(0.3, 0.7) for _ in range(3)], r.uniform(0.5, 1.0), r.uniform(0.08, 0.15)
            u += a * torch.exp(-sum((x[d] - c[d]) ** 2 for d in range(3)) / (2 * w * w))
        if case["path"] == "sipg":
            u = u * torch.sin(math.pi * x[0]) * torch.sin(math.pi * x[1]) * torch.sin(math.pi * x[2])
        out.append(u.reshape(-1))
    return out


def _dt(case):
    gap = float(np.min(np.diff(_gll(case["n"])[0])))
    return (0.2 if case["path"] == "sipg" else 0.1) * gap / max(case["mx"], case["my"], case["mz"])


def _solve(case, seed):
    """Mesh, background, workspace and state of one solve."""
    wt = _wt()
    f32 = case["dtype"] == "f32"
    sipg = case["path"] == "sipg"
    mesh = wt.Mesh.warped_uniform_hex(_ctx(), case["n"], (case["mx"], case["my"], case["mz"]), 0.0, 1.0, case["warp"],
                                      outer_tag=0 if sipg else wt.SOMMERFELD_BDRY_TAG,
                                      precision=wt.WT_F32 if f32 else wt.WT_F64)
    ws = wt.make_wave3d_workspace(mesh)
    if case["eps_ko"]:
        ws.mu
    s = {"case": case, "mesh": mesh, "ws": ws, "dt": _dt(case)}
    if case["path"] not in ("sipg", "strong"):
        s["coef"] = wt.sample_background3d(mesh, wt.BG_ADM_PERTURBED, _adm(seed))
        s["bc"] = wt.make_bc3d([wt.BC_FULL_DIRICHLET if case["bc"] == "full_dirichlet" else wt.BC_SOMMERFELD] * 6)
    a, b = _fields(case, seed, "cuda")
    if f32 and case["path"] in ("rk4", "batch"):
        s["u"], s["v"] = mesh.empty(), mesh.empty()
        wt.state_from_f64(ws, a, b, s["u"], s["v"])
    else:
        s["u"], s["v"] = a.to(mesh.dtype), b.to(mesh.dtype)
    if case["path"] in ("rhs", "strong"):
        s["du"], s["dv"] = mesh.empty(), mesh.empty()
    if case["path"] == "host":
        s["u"], s["v"] = s["u"].cpu().pin_memory(), s["v"].cpu().pin_memory()
    return s


def _member_case(case, n, e):
    return {**case, "n": n, "mx": e, "my": e, "mz": e, "warp": 0.05, "path": "batch"}


def prepare(case, seed):
    if case["path"] != "batch":
        return _solve(case, seed)
    solves = [_solve(_member_case(case, n, e), seed * 100 + k) for k, (n, e) in enumerate(_members(case))]
    batch = _wt().Batch(_ctx())
    for s in solves:
        batch.add(s["u"], s["v"], s["coef"], s["ws"], s["dt"], s["bc"])
    return {"case": case, "batch": batch, "solves": solves}


def run(s):
    wt, c = _wt(), s["case"]
    path = c["path"]
    if path == "batch":
        s["batch"].step(c["steps"])
        return [[m["u"], m["v"]] for m in s["solves"]]
    u, v, ws = s["u"], s["v"], s["ws"]
    if path == "rk4":
        wt.step_rk4_curved(u, v, s["coef"], ws, s["dt"], c["steps"], c["eps_ko"], s["bc"], c["metric"])
    elif path == "tsit5":
        wt.step_erk_curved(u, v, s["coef"], ws, s["dt"], c["steps"], wt.ERK_TSIT5, c["eps_ko"], s["bc"], c["metric"])
    elif path == "rhs":
        return list(wt.wave3d_curved_rhs(s["du"], s["dv"], u, v, s["coef"], ws, c["eps_ko"], s["bc"], c["metric"]))
    elif path == "host":
        e = np.zeros(c["samples"])
        wt.evolve_curved_host(u, v, s["coef"], ws, s["dt"], c["steps"], c["samples"], c["eps_ko"], s["bc"],
                              c["metric"], e)
        return [u, v, e]
    elif path == "sipg":
        wt.step_rk4_sipg(u, v, ws, s["dt"], c["steps"], tau=1.5 * (c["n"] - 1) ** 2, eps_KO=c["eps_ko"])
    elif path == "strong":
        return wt.wave_strong_rhs_mesh(s["du"], u, v, ws)
    return [u, v]


# ---- what one pass cannot do without -----------------------------------------------------


def work(case):
    """Every stage of a step needs the whole state of the stage before it, so a pass's inputs are read once per
    right-hand side: state, coefficients and metric terms in, the stage's result out."""
    if case["path"] == "batch":
        parts = [work({**_member_case(case, n, e), "path": "rk4"}) for n, e in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, w = case["n"], 8 if case["dtype"] == "f64" else 4
    nodes = n ** 3 * case["mx"] * case["my"] * case["mz"]
    path, ko = case["path"], bool(case["eps_ko"])
    if path == "sipg":  # u, ut -> k, with the low-storage stage update (y, accumulator, stage)
        words, flops = 8, 12 * n + 40
    elif path == "strong":  # u (ut on faces) -> utt; 6 metric products and 3 first-derivative weights per node
        words, flops = 11, 18 * n + 40
    else:  # 10 background and 10 metric words; RK4 state words as a low-storage step moves them, else in and out
        words, flops = 20 + (8.5 if path in ("rk4", "host") else 4), 48 * n + 150
    if ko:
        flops += 2 * 3 * 6 * 2 * n
    rhs = {"rk4": 4, "host": 4, "sipg": 4, "tsit5": 6}.get(path, 1) * case["steps"] * case["samples"]
    if path not in ("rhs", "strong"):
        total = words * w * nodes * rhs
    else:
        total = words * w * nodes
    if path == "host":  # an energy (state, 8 coefficients, metric) and a copy out of the state per sample
        total += (2 + 18 + 2) * w * nodes * case["samples"]
    return {"bytes": total, "flops": flops * nodes * rhs}


# ---- the same in plain torch, 64 bits ----------------------------------------------------


class _Plain:
    """The discretisation on the (warped) cube; fields are [ez, ey, ex, k, j, i]."""

    def __init__(self, case, dev):
        self.c, self.n, self.dev = case, case["n"], dev
        self.m = (case["mx"], case["my"], case["mz"])
        _, h, g = _gll(self.n)
        self.H = [float(v) for v in h]
        self.h = torch.tensor(h, dtype=torch.float64, device=dev)
        self.G = torch.tensor(g, dtype=torch.float64, device=dev)
        self.shape = (self.m[2], self.m[1], self.m[0], self.n, self.n, self.n)
        s = _axes(case, dev)
        sn, cs = [torch.sin(2 * math.pi * a) for a in s], [torch.cos(2 * math.pi * a) for a in s]
        tp, A = 2 * math.pi, case["warp"]
        dP = [tp * cs[0] * sn[1] * sn[2], tp * sn[0] * cs[1] * sn[2], tp * sn[0] * sn[1] * cs[2]]
        self.J = [[((1.0 if a == b else 0.0) + A * dP[b]) / self.m[b] for b in range(3)] for a in range(3)]
        del sn, cs, dP
        J = self.J
        cof = [[J[(a + 1) % 3][(b + 1) % 3] * J[(a + 2) % 3][(b + 2) % 3] -
                J[(a + 1) % 3][(b + 2) % 3] * J[(a + 2) % 3][(b + 1) % 3] for b in range(3)] for a in range(3)]
        self.det = J[0][0] * cof[0][0] + J[0][1] * cof[0][1] + J[0][2] * cof[0][2]
        self.inv = [[cof[a][al] / self.det for a in range(3)] for al in range(3)]  # inv[al][a] = d xi_al / d x_a
        self.sdiag = [self.inv[d][d][..., 0, 0, 0][..., None, None, None] for d in range(3)]
        self.mu = None

    def d(self, u, ax):
        """Reference derivative along axis ax of every element."""
        if ax == 0:
            return u @ self.G.T
        if ax == 1:
            return torch.matmul(self.G, u)
        sh = u.shape
        return torch.matmul(self.G, u.reshape(sh[:4] + (self.n * self.n,))).reshape(sh)

    def metric(self):
        """Curl-form metric terms of the coordinates relative to each element's first node."""
        x = [a - a[..., :1, :1, :1] for a in _coords(self.c, self.dev)]
        dx = [[self.d(x[a], b) for b in range(3)] for a in range(3)]
        self.Ja = [[None] * 3 for _ in range(3)]
        for q in range(3):
            l, m = (q + 1) % 3, (q + 2) % 3
            C = [0.5 * (x[l] * dx[m][b] - x[m] * dx[l][b]) for b in range(3)]
            for al in range(3):
                b1, b2 = (al + 1) % 3, (al + 2) % 3
                self.Ja[al][q] = self.d(C[b2], b1) - self.d(C[b1], b2)

    def background(self, p):
        x = _coords(self.c, self.dev)
        tp = 2 * math.pi
        al = 1 + p[0] * torch.sin(tp * x[0])
        b = [p[1] * torch.cos(tp * a) for a in x]
        e = p[2] * torch.exp(-sum((x[d] - p[4 + d]) ** 2 for d in range(3)) / p[3])
        g = [1 + e * (1 + 0.5 * p[7]), 0.5 * e * p[8], 0.5 * e * p[9], 1 + e * (1 + 0.5 * p[10]), 0.5 * e * p[11],
             1 + e * (1 + 0.5 * p[12])]
        det = g[0] * (g[3] * g[5] - g[4] ** 2) - g[1] * (g[1] * g[5] - g[4] * g[2]) + g[2] * (g[1] * g[4] - g[3] * g[2])
        sg = torch.sqrt(det)
        up = [g[3] * g[5] - g[4] ** 2, g[2] * g[4] - g[1] * g[5], g[1] * g[4] - g[2] * g[3], g[0] * g[5] - g[2] ** 2,
              g[1] * g[2] - g[0] * g[4], g[0] * g[3] - g[1] ** 2]
        self.sg, self.up = sg, [v / det for v in up]
        self.a, self.b, self.K = al / sg, b, [al * sg * v / det for v in up]

    def face(self, u, ax, hi):
        return u.select(5 - ax, self.n - 1 if hi else 0)

    def across(self, u, ax, hi):
        """The neighbour's trace on a face, 0 on the outer boundary, and whether there is a neighbour."""
        t = self.face(u, ax, not hi)
        e = 2 - ax
        out, has = torch.zeros_like(t), torch.zeros(t.shape[:3] + (1, 1), dtype=torch.bool, device=self.dev)
        k = self.m[ax]
        to, fr = (slice(0, k - 1), slice(1, k)) if hi else (slice(1, k), slice(0, k - 1))
        at = [slice(None)] * 3
        src = list(at)
        at[e], src[e] = to, fr
        out[tuple(at)] = t[tuple(src)]
        has[tuple(at)] = True
        return out, has

    def jump(self, u, ax, hi):
        t, has = self.across(u, ax, hi)
        return torch.where(has, t - self.face(u, ax, hi), torch.zeros_like(t))

    def grad(self, u):
        g = []
        for c in range(3):
            acc = 0
            for al in range(3):
                J = self.Ja[al][c]
                acc = acc + 0.5 * self.d(J * u, al) + 0.5 * J * self.d(u, al)
            for al in range(3):
                for hi in (0, 1):
                    v = self.face(acc, al, hi)
                    v += (1 if hi else -1) * self.face(self.Ja[al][c], al, hi) * self.jump(u, al, hi) / (2 * self.H[0])
            g.append(acc / self.det)
        return g

    def div(self, F):
        acc = 0
        for al in range(3):
            w = sum(self.Ja[al][c] * F[c] for c in range(3))
            acc = acc + 0.5 * self.d(w, al)
            for c in range(3):
                acc = acc + 0.5 * self.Ja[al][c] * self.d(F[c], al)
        for al in range(3):
            for hi in (0, 1):
                v = self.face(acc, al, hi)
                for c in range(3):
                    v += (1 if hi else -1) * self.face(self.Ja[al][c], al, hi) * self.jump(F[c], al, hi) / (2 * self.H[0])
        return acc / self.det

    def apply_D(self, u, ax):
        s = self.sdiag[ax]
        out = s * self.d(u, ax)
        for hi in (0, 1):
            v = self.face(out, ax, hi)
            v += (1 if hi else -1) * s[..., 0] * self.jump(u, ax, hi) / (2 * self.H[0])
        return out

    def ko(self, u, eps):
        if self.mu is None:
            i = torch.arange(self.n, device=self.dev)
            e = torch.arange(self.m[0] * self.m[1] * self.m[2], device=self.dev).reshape(self.shape[:3])
            odd = (i + i[:, None] + i[:, None, None] + e[..., None, None, None]) % 2
            v = torch.where(odd == 1, 1.0, -1.0).to(torch.float64)
            for _ in range(30):
                v = self.apply_D(self.apply_D(v, 0), 0)
                mu2 = float(v.norm())
                v = v / mu2
            self.mu = math.sqrt(mu2)
        out = 0
        for ax in range(3):
            w = u
            for _ in range(6):
                w = self.apply_D(w, ax)
            out = out + w
        return eps * self.mu ** -5 * out

    def rhs(self, P, Q):
        g, b, K = self.grad(P), self.b, self.K
        F = [b[0] * Q + K[0] * g[0] + K[1] * g[1] + K[2] * g[2], b[1] * Q + K[1] * g[0] + K[3] * g[1] + K[4] * g[2],
             b[2] * Q + K[2] * g[0] + K[4] * g[1] + K[5] * g[2]]
        dP = b[0] * g[0] + b[1] * g[1] + b[2] * g[2] + self.a * Q
        dQ = self.div(F)
        del F
        if self.c["eps_ko"]:
            dP = dP + self.ko(P, self.c["eps_ko"])
            dQ = dQ + self.ko(Q, self.c["eps_ko"])
        for ax in range(3):
            for hi in (0, 1):
                at = [slice(None)] * 3
                at[2 - ax] = self.m[ax] - 1 if hi else 0
                at = tuple(at)
                f = lambda u: self.face(u, ax, hi)[at]  # noqa: E731
                p, q = (1, 2) if ax == 0 else (0, 2) if ax == 1 else (0, 1)
                t, r = [f(self.J[a][p]) for a in range(3)], [f(self.J[a][q]) for a in range(3)]
                so = (1 if hi else -1) * (-1 if ax == 1 else 1)
                nf = [so * (t[(a + 1) % 3] * r[(a + 2) % 3] - t[(a + 2) % 3] * r[(a + 1) % 3]) for a in range(3)]
                JF = torch.sqrt(sum(v * v for v in nf))
                nv = [v / JF for v in nf]
                k = [f(v) for v in K]
                Kn = (k[0] * nv[0] ** 2 + k[3] * nv[1] ** 2 + k[5] * nv[2] ** 2 +
                      2 * (k[1] * nv[0] * nv[1] + k[2] * nv[0] * nv[2] + k[4] * nv[1] * nv[2]))
                a0 = f(self.a)
                an = torch.sqrt(a0 * Kn)
                bn = sum(f(b[d]) * nv[d] for d in range(3))
                wt = JF / (self.H[0] * f(self.det))
                if self.c["bc"] == "full_dirichlet":
                    tau = ((an - bn).abs() + (an + bn).abs()) * wt
                    self.face(dP, ax, hi)[at] -= tau * f(P)
                    self.face(dQ, ax, hi)[at] -= tau * f(Q)
                else:
                    q_ = sum(nv[d] * f(g[d]) for d in range(3))
                    self.face(dQ, ax, hi)[at] -= (an + bn).abs() * wt * (f(Q) + (bn + an) / a0 * q_)
        return dP, dQ

    def energy(self, P, Q):
        g, u = self.grad(P), self.up
        dens = Q * Q / self.sg + self.sg * (u[0] * g[0] ** 2 + u[3] * g[1] ** 2 + u[5] * g[2] ** 2 +
                                            2 * (u[1] * g[0] * g[1] + u[2] * g[0] * g[2] + u[4] * g[1] * g[2]))
        h = self.h
        return float((dens * self.det.abs() * h * h[:, None] * h[:, None, None]).sum()) / 2

    def sipg(self, u, v):
        """u_t = v, v_t = L u (Dirichlet 0 outside), both with dissipation."""
        tau, out = 1.5 * (self.n - 1) ** 2, 0
        for ax in range(3):
            s = float(self.m[ax])
            D = s * self.d(u, ax)
            out = out + s * self.d(D, ax)
            for hi in (0, 1):
                r, nh = (self.n - 1 if hi else 0), (1 if hi else -1)
                t, has = self.across(u, ax, hi)
                dt, _ = self.across(D, ax, hi)
                du = self.face(u, ax, hi) - t
                dG = torch.where(has, self.face(D, ax, hi) - dt, torch.zeros_like(t))
                al = torch.where(has, 0.5, 1.0)
                w = self.face(out, ax, hi)
                w += (-tau * s * s * du - 0.5 * nh * s * dG) / self.H[0]
                sh = [1] * 6
                sh[5 - ax] = self.n
                out += nh * s * s * (self.G[r] / self.h).view(sh) * (al * du).unsqueeze(5 - ax)
        eps = self.c["eps_ko"]
        return (v + self.ko(u, eps), out + self.ko(v, eps)) if eps else (v, out)

    def strong(self, u, v):
        inv, tau = self.inv, float((self.n - 1) ** 2)
        du = [self.d(u, a) for a in range(3)]
        dp = [sum(inv[al][a] * du[al] for al in range(3)) for a in range(3)]
        out = 0
        for al in range(3):
            for be in range(3):
                out = out + sum(inv[al][a] * inv[be][a] for a in range(3)) * self.d(du[min(al, be)], max(al, be))
                out = out + sum(inv[al][a] * self.d(inv[be][a], al) for a in range(3)) * du[be]
        for ax in range(3):
            nrm = torch.sqrt(sum(inv[ax][a] ** 2 for a in range(3)))
            for hi in (0, 1):
                f = lambda w: self.face(w, ax, hi)  # noqa: E731
                t, has = self.across(u, ax, hi)
                dn = (1 if hi else -1) * sum(f(inv[ax][a]) * f(dp[a]) for a in range(3)) / f(nrm)
                w = f(nrm) / self.H[0]
                f(out).sub_(torch.where(has, w * dn + tau * w * (f(u) - t), w * (f(v) + dn)))
        return out


_TSIT5 = ([[], [0.161], [-0.008480655492356989, 0.335480655492357],
           [2.897153057105493, -6.359448489975075, 4.3622954328695815],
           [5.325864828439257, -11.748883564062828, 7.4955393428898365, -0.09249506636175525],
           [5.86145544294642, -12.92096931784711, 8.159367898576159, -0.071584973281401, -0.028269050394068383]],
          [0.09646076681806523, 0.01, 0.4798896504144996, 1.379008574103742, -3.290069515436081, 2.324710524099774])
_RK4 = ([[], [0.5], [0.0, 0.5], [0.0, 0.0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6])


def _steps(f, u, v, dt, tableau, count):
    A, b = tableau
    for _ in range(count):
        ks = []
        for row in A:
            x = u + dt * sum(a * k[0] for a, k in zip(row, ks) if a) if any(row) else u
            y = v + dt * sum(a * k[1] for a, k in zip(row, ks) if a) if any(row) else v
            ks.append(f(x, y))
        u = u + dt * sum(a * k[0] for a, k in zip(b, ks))
        v = v + dt * sum(a * k[1] for a, k in zip(b, ks))
        del ks
    return u, v


def _exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = _Plain(case, dev)
    u, v = (a.reshape(f.shape) for a in _fields(case, seed, dev))
    path, dt = case["path"], _dt(case)
    if case["dtype"] == "f32" and path not in ("rk4", "batch"):  # those two start from the 64-bit state itself
        u, v = u.float().double(), v.float().double()
    if path == "strong":
        return f.strong(u, v).reshape(-1)
    if path == "sipg":
        return [a.reshape(-1) for a in _steps(f.sipg, u, v, dt, _RK4, case["steps"])]
    f.metric()
    f.background(_adm(seed))
    if path == "rhs":
        return [a.reshape(-1) for a in f.rhs(u, v)]
    if path == "host":
        e = []
        for _ in range(case["samples"]):
            u, v = _steps(f.rhs, u, v, dt, _RK4, case["steps"])
            e.append(f.energy(u, v))
        return [u.reshape(-1), v.reshape(-1), np.array(e)]
    return [a.reshape(-1) for a in _steps(f.rhs, u, v, dt, _TSIT5 if path == "tsit5" else _RK4, case["steps"])]


def exact(case, seed):
    if case["path"] == "batch":
        return [_exact(_member_case(case, n, e), seed * 100 + k) for k, (n, e) in enumerate(_members(case))]
    return _exact(case, seed)
