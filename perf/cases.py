"""Workloads of the framework's entry points: right-hand sides, RK4 steps, batches, source-mode runs
and adjoint sweeps over the range of meshes, degrees, coefficients and options that programs use.

A case is a dict of plain values:
  kind      rhs      Workspace.rhs (edg_rhs!) on CUDA tensors
            rhs_host edg_rhs_ on host arrays, as the reference's callers hold them
            rk4      `steps` RK4 steps (Workspace.rk4_steps) from a kept state on CUDA tensors
            batch    `steps` RK4 steps of `count` mixed instances (Batch.rk4_steps)
            source   Workspace.run_source: steps with receivers, energy series, slices
            adjoint  Workspace.rk4_adjoint over `steps` steps, with the coefficient gradients
  N, q      mesh N x N and degree of u;  mixed: the degree of v is q - 1
  mode      mms, initial_value or source
  coef      paper (the smooth weak ones), const, vary (10 % around the constants), cells (4 x 4 jumping)
  flux, bnd flux name; legacy boundary kind, or "open" (one absorbing side, three walls), "all4"
  count, mix     instances of a batch and the seed of their sizes and options
  solver, cheb   mass solver; Chebyshev counts per element or common to the mesh
  state     smooth (long waves), front (steep front over long waves), short (every element steep)
"""
import math

import numpy as np
import torch

BOUNDS = {"open": dict(bot="absorbing_2beta", top="wall", lft="wall", rgt="wall"),
          "all4": dict(bot="dirichlet", top="absorbing", lft="absorbing_2beta", rgt="wall")}
DEFAULT = dict(kind="rk4", N=64, q=4, mixed=False, mode="source", coef="const", flux="alternating", bnd="open",
               solver="chebyshev", cheb="per_element", state="smooth", steps=1, count=1, mix=0)
SIGMA, KAPPA = 0.25, 0.5


def _case(**kw):
    return {**DEFAULT, **kw}


def listed():
    return [
        # one call on the mesh of the regression tests: launch latency
        _case(name="rhs_n10_q3", kind="rhs", N=10, q=3, mixed=True, mode="mms", coef="paper", flux="upwind",
              bnd="absorbing_2beta"),
        # the middle of the convergence tables: smooth coefficients, manufactured solution
        _case(name="rk4_n32_q4_mms", N=32, q=4, mixed=True, mode="mms", coef="paper", flux="upwind",
              bnd="absorbing_2beta", steps=8),
        # the plain source-mode simulation with its receivers and energy series
        _case(name="source_n64_q4", kind="source", N=64, q=4, steps=64),
        # the GPU-scale mesh of the plain method: a steep front over long waves
        _case(name="rk4_n512_q6_front", N=512, q=6, state="front", steps=1),
        # the same path called on host arrays by a host program (copies included)
        _case(name="rhs_host_n256_q6", kind="rhs_host", N=256, q=6, state="front"),
        # jumping coefficients, mixed degrees, four kinds of sides, one-sided faces
        _case(name="rk4_n256_q5_jump", N=256, q=5, mixed=True, mode="initial_value", coef="cells", flux="central",
              bnd="all4", steps=4),
        # coefficients that vary inside the elements (stored inverses), odd mesh
        _case(name="rk4_n201_q6_vary", N=201, q=6, coef="vary", state="front", flux="upwind"),
        # the conjugate-gradient mass solver, odd mesh
        _case(name="rk4_n97_q5_cg", N=97, q=5, flux="upwind", bnd="absorbing", solver="cg", state="front", steps=2),
        # strongly nonlinear everywhere: the mass solve takes its largest counts
        _case(name="rhs_n300_q7_short", kind="rhs", N=300, q=7, state="short"),
        # the reference's own policy of one Chebyshev count for all elements, low degree
        _case(name="rk4_n333_q2_common", N=333, q=2, flux="upwind", cheb="common_max", state="front", steps=2),
        # a parameter study: mixed instances advanced together
        _case(name="batch_16", kind="batch", N=96, q=7, coef="cells", count=16, mix=4, steps=4),
        # one checkpoint segment's worth of a misfit gradient
        _case(name="adjoint_n128_q4", kind="adjoint", N=128, q=4, coef="cells", flux="upwind",
              bnd="absorbing_2beta", steps=8),
    ]


def draw(rng):
    kind = rng.choice(["rhs", "rk4", "rk4", "rk4", "rhs_host", "batch", "source", "adjoint"])
    c = _case(kind=kind, mixed=rng.random() < 0.4, flux=rng.choice(["upwind", "central", "alternating"]),
              bnd=rng.choice(["open", "all4", "absorbing_2beta", "absorbing", "dirichlet", "wall"]))
    q = rng.randint(2, 7)
    top = {"rhs": 400, "rk4": 320, "rhs_host": 256, "batch": 96, "source": 80, "adjoint": 128}[kind]
    if kind != "batch" and q >= 6:
        top = int(top * 0.8)
    N = int(round(math.exp(rng.uniform(math.log(8), math.log(top)))))
    c["q"] = q
    c["coef"] = rng.choice(["const", "cells", "vary", "paper"])
    c["mode"] = rng.choice(["source", "initial_value", "mms"])
    c["state"] = rng.choice(["smooth", "front", "front", "short"] if kind in ("rhs", "rhs_host", "rk4") else
                            ["smooth", "front"])
    c["steps"] = {"rk4": rng.randint(1, 3), "batch": rng.randint(2, 6), "source": rng.randint(16, 48),
                  "adjoint": rng.randint(2, 6)}.get(kind, 1)
    if kind in ("batch", "adjoint"):
        c["coef"], c["mode"] = "cells", "source"
        c["count"] = rng.randint(4, 16) if kind == "batch" else 1
        c["mix"] = rng.randint(0, 999) if kind == "batch" else 0
    if kind == "source":
        c["mode"] = "source"
    if kind == "adjoint":
        c["q"] = min(q, 5)
    if kind in ("rhs", "rk4"):
        c["solver"] = rng.choice(["chebyshev", "chebyshev", "chebyshev", "cg"])
        if c["solver"] == "chebyshev":
            c["cheb"] = rng.choice(["per_element", "per_element", "common_max"])
    if c["coef"] == "cells":
        N = max(8, 4 * (N // 4))                    # the 4 x 4 cells are unions of elements
        if c["mode"] == "mms":
            c["mode"] = "initial_value"             # a manufactured solution needs continuous coefficients
    c["N"] = N
    return c


# ---------------------------------------------------------------------------- problem data

def _trig(a, b):
    """Coefficient functions of numpy arrays: 1 + s cos(pi x) cos(pi y) and its derivatives."""
    pi = math.pi
    return (lambda x, y: a + b * np.cos(pi * x) * np.cos(pi * y),
            lambda x, y: -b * pi * np.sin(pi * x) * np.cos(pi * y),
            lambda x, y: -b * pi * np.cos(pi * x) * np.sin(pi * y))


def _coefs(case, seed):
    """(c, c_x, c_y, alpha, alpha_x, alpha_y, beta) as functions, or the tables of 4 x 4 cells; the largest
    c and beta."""
    pi, kind = math.pi, case["coef"]
    if kind == "cells":
        r = np.random.default_rng(1000 + seed)
        weak = case["kind"] == "adjoint"            # the explicit step of the adjoint workloads wants small alpha
        c = r.uniform(0.8, 1.25, (4, 4)) if weak else r.uniform(0.5, 2.0, (4, 4))
        al = 10.0 ** r.uniform(-6, -5 if weak else -3, (4, 4))
        be = r.uniform(0.5, 4.0 if weak else 10.0, (4, 4))
        return (c, al, be), float(c.max()), float(be.max())
    s = {"paper": 0.1, "vary": 0.1, "const": 0.0}[kind]
    a0, a1, b0 = {"paper": (1e-5, 1e-6, 1e-4), "vary": (1e-6, 1e-7, 8.0), "const": (1e-6, 0.0, 8.0)}[kind]
    be = lambda x, y: b0 * (1 + s * np.sin(pi * x) * np.sin(pi * y))  # noqa: E731
    return (*_trig(1.0, s), *_trig(a0, a1), be), 1.0 + s, b0 * (1 + s)


def _profile(seed):
    """Initial displacement: three Gaussians of amplitude 1e-3 and their derivatives."""
    r = np.random.default_rng(2000 + seed)
    cen, wid, amp = r.uniform(0.2, 0.8, (3, 2)), r.uniform(0.05, 0.1, 3), 1e-3 * r.uniform(-1, 1, 3)

    def f(d):
        def g(x, y):
            out = 0.0
            for (x0, y0), w, a in zip(cen, wid, amp):
                X, Y = np.asarray(x) - x0, np.asarray(y) - y0
                e = a * np.exp(-(X * X + Y * Y) / (w * w))
                out = out + {"": e, "x": -2 * X / w ** 2 * e, "y": -2 * Y / w ** 2 * e,
                             "xx": (4 * X * X / w ** 4 - 2 / w ** 2) * e,
                             "yy": (4 * Y * Y / w ** 4 - 2 / w ** 2) * e}[d]
            return out
        return g
    return dict(u0=f(""), u0_x=f("x"), u0_y=f("y"), u0_xx=f("xx"), u0_yy=f("yy"))


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _basis(n, x):
    """Orthonormal Legendre values and derivatives of n modes at the points x: two (len(x), n) arrays."""
    L = np.polynomial.legendre
    s = np.sqrt((2 * np.arange(n) + 1) / 2)
    P = np.stack([L.legval(x, np.eye(n)[d]) for d in range(n)], 1) * s
    D = np.stack([L.legval(x, L.legder(np.eye(n)[d])) if d else np.zeros(len(x)) for d in range(n)], 1) * s
    return P, D


def _state(case, seed):
    """Modal coefficients [j, k, a, b] (row, column, mode in y, mode in x) of the state, on the device.
    v stays within |2 beta v| <= 0.58, the range of the steepened runs."""
    N, nu = case["N"], case["q"] + 1
    nv = nu - int(case["mixed"])
    r = np.random.default_rng(seed)
    bmax = _coefs(case, seed)[2]
    amp = min(0.58 / (2 * bmax), 5.0)
    z, w = np.polynomial.legendre.leggauss(nu + 2)
    h, dev = 1.0 / N, _dev()
    T = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    pts = T((np.arange(N)[:, None] + 0.5 + 0.5 * z[None, :]) * h)
    X, Y = pts[None, :, None, :], pts[:, None, :, None]
    m = r.integers(1, 5, (3, 2))
    ph, wt = r.uniform(0, 2 * math.pi, (3, 2)), r.uniform(0.2, 1.0, 3)
    wave = sum(float(wt[i] / 3) * torch.sin(2 * math.pi * int(m[i, 0]) * X + float(ph[i, 0]))
               * torch.cos(2 * math.pi * int(m[i, 1]) * Y + float(ph[i, 1])) for i in range(3))
    if case["state"] == "smooth":
        v = 0.02 * amp * wave
    elif case["state"] == "front":
        R = float(r.uniform(0.3, 0.5))
        v = amp * (0.999 * torch.tanh((torch.hypot(X - 0.15, Y - 0.5) - R) / h) + 1e-3 * wave)
    else:
        v = amp * torch.sin(2 * math.pi / h * X) * torch.sin(2 * math.pi / h * Y + float(ph[0, 0]))
        v = 0.95 * v + 0.05 * amp * wave
    u = 1e-4 * wave.flip(0) if case["state"] != "smooth" else 1e-3 * wave.flip(1)

    def modes(f, n):
        Pw = T(_basis(n, z)[0] * w[:, None])
        return torch.einsum("ra,jkrs,sb->jkab", Pw, f, Pw)
    return modes(u, nu), modes(v, nv)


def _flat(x):
    """[j, k, a, b] to the library's bytes (j fastest) as a flat tensor."""
    return x.permute(3, 2, 1, 0).reshape(-1).contiguous()


def _host(x):
    return np.asfortranarray(x.cpu().numpy())


def _bound(case):
    return BOUNDS.get(case["bnd"], case["bnd"])


def _t0(seed):
    return float(np.random.default_rng(3000 + seed).uniform(0.2, 0.6))


def _dt(case, seed):
    return (1.0 / case["N"]) / (10.0 * _coefs(case, seed)[1] * case["q"] ** 2)


def _parts(case, seed):
    """The instances of a batch as cases of their own, with the seeds of their data (the mix of sizes and
    options is the case's)."""
    r = np.random.default_rng(case["mix"])
    out = []
    for i in range(case["count"]):
        q = int(r.integers(2, case["q"] + 1))
        N = 4 * int(r.integers(2, max(3, case["N"] // 4) + 1))
        kinds = [str(k) for k in r.choice(["open", "all4", "absorbing", "wall"], 1)]
        out.append(({**case, "kind": "rk4", "q": q, "N": N, "mixed": bool(r.integers(0, 2)), "bnd": kinds[0],
                     "flux": str(r.choice(["upwind", "central", "alternating"]))}, seed + 17 * i))
    return out


def _workspace(case, seed):
    import edg_westervelt_gb300 as W
    co = _coefs(case, seed)[0]
    if case["coef"] == "cells":
        co = W.cell_coefficients(*co)
    elif case["coef"] == "const":
        co = W.constant_coefficients(c=1.0, alpha=1e-6, beta=8.0)
    else:
        co = W.Coefficients(*co)
    kw = dict(initial_profile=_profile(seed)) if case["mode"] == "initial_value" else {}
    pre, geo = W.precompute(case["q"], case["N"], mixed=bool(case["mixed"]), flux=case["flux"], sigma=SIGMA,
                            kappa=KAPPA, boundary=_bound(case), coefficients=co, mode=case["mode"],
                            mass_solver=case["solver"], target="device", **kw)
    return W.Workspace(pre, case["N"], cheb_steps=case["cheb"]), pre, geo


RECEIVERS = ((0.45, 0.5), (0.7, 0.5), (0.85, 0.5))
RECORD, SLICE_Y = 20, 0.5


def _locate(s, N):
    i = min(max(int(math.ceil(s * N)), 1), N)
    return i - 1, min(max(2 * (s * N - (i - 1)) - 1, -1.0), 1.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        import edg_westervelt_gb300 as W
        parts = _parts(case, seed)
        S = dict(kind=kind, ws=[_workspace(c, s)[0] for c, s in parts], steps=case["steps"],
                 t0=[_t0(s) for _, s in parts], dt=[_dt(c, s) for c, s in parts])
        start = [_state(c, s) for c, s in parts]
        S["u0"], S["v0"] = [_flat(u) for u, _ in start], [_flat(v) for _, v in start]
        S["u"], S["v"] = [x.clone() for x in S["u0"]], [x.clone() for x in S["v0"]]
        S["batch"] = W.Batch(S["ws"])
        return S
    ws, pre, geo = _workspace(case, seed)
    u, v = _state(case, seed)
    S = dict(kind=kind, ws=ws, pre=pre, N=case["N"], t0=_t0(seed), dt=_dt(case, seed), steps=case["steps"])
    if kind in ("rhs", "rk4"):
        # device-resident states, the library on the program's stream
        S["stream"] = torch.cuda.Stream()
        ws.set_stream(S["stream"].cuda_stream)
        S["u0"], S["v0"] = _flat(u), _flat(v)
        S["u"], S["v"] = torch.empty_like(S["u0"]), torch.empty_like(S["v0"])
        return S
    S["u0"], S["v0"] = _host(u), _host(v)
    if kind == "adjoint":
        lam = _state({**case, "state": "smooth"}, seed + 5)
        S["lu"], S["lv"] = (_host(x / x.abs().max()) for x in lam)
    if kind == "source":
        S["u"], S["v"] = S["u0"].copy(order="F"), S["v0"].copy(order="F")
        nv, N = pre["qv1"], case["N"]
        row = lambda r: _basis(nv, np.array([r]))[0][0]  # noqa: E731
        at = [(_locate(y, N), _locate(x, N)) for x, y in RECEIVERS]
        S["rec"] = ([(a[0], b[0]) for a, b in at], np.stack([row(a[1]) for a, _ in at]),
                    np.stack([row(b[1]) for _, b in at]))
        j, eta = _locate(SLICE_Y, N)
        S["slice"], S["err"] = (j, row(eta)), (geo["err_c2"], geo["err_beta"])
    return S


def run(S):
    kind = S["kind"]
    if kind == "batch":
        for d, s in zip(S["u"] + S["v"], S["u0"] + S["v0"]):
            d.copy_(s)
        torch.cuda.current_stream().synchronize()        # the batch runs on streams of its own
        S["batch"].rk4_steps(S["u"], S["v"], S["t0"], S["dt"], S["steps"])
        return S["u"] + S["v"]
    ws = S["ws"]
    if kind == "rhs":
        with torch.cuda.stream(S["stream"]):
            ws.rhs(S["u0"], S["v0"], S["t0"], S["u"], S["v"])
        return S["u"], S["v"]
    if kind == "rk4":
        with torch.cuda.stream(S["stream"]):
            S["u"].copy_(S["u0"])
            S["v"].copy_(S["v0"])
            ws.rk4_steps(S["u"], S["v"], S["t0"], S["dt"], S["steps"])
        return S["u"], S["v"]
    if kind == "rhs_host":
        import edg_westervelt_gb300 as W
        return W.edg_rhs_(ws, S["u0"], S["v0"], S["t0"], S["N"], 1.0 / S["N"], S["pre"])
    if kind == "adjoint":
        return ws.rk4_adjoint(S["u0"], S["v0"], S["t0"], S["dt"], S["steps"], S["lu"], S["lv"], every=4, params=True)
    np.copyto(S["u"], S["u0"])
    np.copyto(S["v"], S["v0"])
    done, recv, energy, vmax, ndmin, slices, snaps = ws.run_source(
        S["u"], S["v"], S["t0"], S["dt"], S["steps"], RECORD, *S["rec"], *S["slice"], [S["steps"]], *S["err"])
    return dict(u=S["u"], v=S["v"], recv=recv, energy=energy, vmax=vmax, ndmin=ndmin, slices=slices, snap=snaps[0])


# ---------------------------------------------------------------------------- work

def _sizes(case):
    nu = case["q"] + 1
    nv = nu - int(case["mixed"])
    qh = max(math.ceil(3 * (nv - 1) / 2) + 1, nu)
    return nu, nv, qh, case["N"] ** 2


def _work(case):
    """Bytes: the state read and written once, the coefficient data read once. Operations: the sum
    factorised volume terms, traces, lifts, the u-solve by the eigenbasis (constants and cells) or the
    stored inverse, one forming of the mass weights and two applications of the mass matrix a stage."""
    nu, nv, qh, E = _sizes(case)
    fast = case["coef"] in ("const", "cells")
    data = qh * qh + nv * nv + (3 if fast else nu * nu * (nu * nu + 1) / 2 + 2 * nu * nu + 12 * nu)
    vol = 8 * nu * nv * nu if fast else 16 * nu ** 3 + 8 * nu * nv * (nu + nv)
    solve = 8 * nu ** 3 / 2 if fast else 2 * nu ** 4
    face = 4 * (4 * nv * nu + 4 * nu * nu + 12 * nu)
    mass = (2 * qh * nv * (nv + qh) + 2 * 4 * qh * nv * (nv + qh)) / 2 + 20 * nv * nv
    stages = {"rhs": 1, "rhs_host": 1, "adjoint": 3 * 4 * case["steps"]}.get(case["kind"], 4 * case["steps"])
    return {"bytes": 8.0 * E * (2 * (nu * nu + nv * nv) + data), "flops": float(E) * stages * (vol + solve + face + mass)}


def work(case):
    if case["kind"] != "batch":
        return _work(case)
    w = [_work(c) for c, _ in _parts(case, 1)]
    return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------- the method in plain torch

class _Dense:
    """The semi-discrete right-hand side by dense element operators and direct solves, in 64 bits."""

    def __init__(self, case, seed, grads=False):
        self.case, self.N, dev = case, case["N"], _dev()
        self.nu, self.nv, self.qh, _ = _sizes(case)
        N, nu, nv, qh = self.N, self.nu, self.nv, self.qh
        T = self.T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        z, w = np.polynomial.legendre.leggauss(nu)
        zh, wh = np.polynomial.legendre.leggauss(qh)
        self.z, self.w = z, T(w)
        P, D = _basis(nu, z)
        self.P, self.D = T(P), T(D)
        e, d = _basis(nu, np.array([-1.0, 1.0]))
        self.E, self.E1 = T(e), T(d)
        self.Ph, self.W = T(_basis(nv, zh)[0]), T(np.outer(wh, wh))
        Ph = self.Ph
        self.Phi = torch.einsum("ra,sb->rsab", Ph, Ph).reshape(qh * qh, nv * nv)
        h = 1.0 / N
        self.th2 = 2.0 / h
        cells = np.arange(N)
        xl, xh = (cells[:, None] + 0.5 + 0.5 * z) * h, (cells[:, None] + 0.5 + 0.5 * zh) * h
        self.xl = xl
        co = _coefs(case, seed)[0]
        if case["coef"] == "cells":
            up = lambda a: T(np.repeat(np.repeat(a, N // 4, 0), N // 4, 1))  # noqa: E731
            self.c2, self.al, self.be = up(co[0] ** 2), up(co[1]), up(co[2])
            if grads:
                for x in (self.c2, self.al, self.be):
                    x.requires_grad_(True)
            c2q, alq, beq = (x[:, :, None, None].expand(N, N, nu, nu) for x in (self.c2, self.al, self.be))
            self.beh = self.be[:, :, None, None].expand(N, N, qh, qh)
            face = lambda x: [x[:, :, None].expand(N, N, nu)] * 4  # noqa: E731
            self.fc2, self.fal, self.fbe = face(self.c2), face(self.al), face(self.be)
            self.c2h = self.c2[:, :, None, None]
            div = lambda sx, sy, sxx, syy: (self.c2h * (sxx + syy), None)  # noqa: E731
        else:
            grid = lambda p: (p[None, :, None, :], p[:, None, :, None])  # noqa: E731
            ev = lambda f, X, Y: T(np.broadcast_to(f(X, Y), np.broadcast_shapes(X.shape, Y.shape)) + 0.0 * X + 0.0 * Y)  # noqa: E731
            XQ, high = grid(xl), grid(xh)
            cq, alq, beq = ev(co[0], *XQ), ev(co[3], *XQ), ev(co[6], *XQ)
            c2q = cq * cq
            self.beh = ev(co[6], *high)
            lo, hi = cells[:, None] * h, (cells[:, None] + 1) * h

            def sides(f):   # bottom, top, left, right of every element, at its face points
                return [ev(f, xl[None, :, :], s[:, :, None]) for s in (lo, hi)] + \
                       [ev(f, s[None, :, :], xl[:, None, :]) for s in (lo, hi)]
            self.fc2 = [x * x for x in sides(co[0])]
            self.fal, self.fbe = sides(co[3]), sides(co[6])

            def div(sx, sy, sxx, syy):
                c, cx, cy, a, ax, ay = (ev(f, *high) for f in co[:6])
                return 2 * c * cx * sx + 2 * c * cy * sy + c * c * (sxx + syy), ax * sx + ay * sy + a * (sxx + syy)
        w2 = self.w[:, None] * self.w[None, :]
        self.Cw, self.Aw = c2q * w2, alq * w2
        self.c2q, self.beq = c2q, beq
        XH, YH = xh[None, :, None, :], xh[:, None, :, None]
        self.proj = lambda f: torch.einsum("ra,jkrs,sb->jkab", Ph, self.W * f, Ph)
        self.om = 2 * math.pi * math.sqrt(2.0)
        mode, p2 = case["mode"], 2 * math.pi
        self.mms, self.src = mode == "mms", mode == "source"
        self.jc = None
        self.bd = None
        if self.src:
            self.srcP = self.proj(T(np.exp(-((XH - 0.15) ** 2 + (YH - 0.5) ** 2) / 0.05 ** 2)))
        else:
            if mode == "mms":
                s0 = lambda x, y: np.cos(p2 * x) * np.sin(p2 * y)  # noqa: E731
                sx = lambda x, y: -p2 * np.sin(p2 * x) * np.sin(p2 * y)  # noqa: E731
                sy = lambda x, y: p2 * np.cos(p2 * x) * np.cos(p2 * y)  # noqa: E731
                sxx = syy = lambda x, y: -p2 * p2 * s0(x, y)  # noqa: E731
            else:
                f = _profile(seed)
                s0, sx, sy, sxx, syy = f["u0"], f["u0_x"], f["u0_y"], f["u0_xx"], f["u0_yy"]
            at = lambda f: T(f(XH + 0 * YH, YH + 0 * XH))  # noqa: E731
            cdiv, ddiv = div(at(sx), at(sy), at(sxx), at(syy))
            self.pC = self.proj(cdiv)
            if self.mms:
                self.pS, self.pB, self.pD = self.proj(at(s0)), self.proj(self.beh * at(s0) ** 2), self.proj(ddiv)
            one, zero = np.ones_like(xl), np.zeros_like(xl)
            self.bd = [(T(s0(xl, zero)), T(sy(xl, zero))), (T(s0(xl, one)), T(sy(xl, one))),
                       (T(s0(zero, xl)), T(sx(zero, xl))), (T(s0(one, xl)), T(sx(one, xl)))]
            # the jump of c2 du0/dn across the interior faces (rows j | j+1, columns k | k+1)
            f = np.arange(1, N) * h
            gy = T(sy(xl[None, :, :] + 0 * f[:, None, None], f[:, None, None] + 0 * xl[None, :, :]))
            gx = T(sx(f[None, :, None] + 0 * xl[:, None, :], xl[:, None, :] + 0 * f[None, :, None]))
            self.jc = ((self.fc2[1][:-1] - self.fc2[0][1:]) * gy, (self.fc2[3][:, :-1] - self.fc2[2][:, 1:]) * gx)
        th, tau, lu, lv = {"upwind": (1, 1, 1, 1), "alternating": (1, 0, 0, 0), "central": (0.5, 0, 0, 0)}[case["flux"]]
        self.fl = (th, tau, lu, lv)
        b = _bound(case)
        self.kinds = [b[s] for s in ("bot", "top", "lft", "rgt")] if isinstance(b, dict) else [b] * 4
        K1 = self.D.T @ (self.w[:, None] * self.D)
        I = torch.eye(nu, dtype=torch.float64, device=dev)
        A = torch.kron(K1, I) + torch.kron(I, K1)
        A[0, 0] += 1.0
        self.A1 = A

    def boundary(self, s, t, c2, al, be, v, gu, gv):
        """Flux slots of a physical side: gu, gv the outward normal derivatives, c2, al, be, v at its points."""
        ct, st = (math.cos(self.om * t), math.sin(self.om * t)) if self.mms else (0.0, 0.0)
        sgn = -1.0 if s in (0, 2) else 1.0
        c = torch.sqrt(c2)
        gue = gve = vex = torch.zeros_like(v)
        if self.bd is not None:
            sp, spn = self.bd[s]
            gue, gve, vex = sgn * (ct - 1.0) * spn, -sgn * self.om * st * spn, -self.om * st * sp
        kind = self.kinds[s]
        if kind == "wall":
            g2 = c2 * gue + al * gve
            return g2, -(KAPPA / c) * (c2 * gu + al * gv - g2)
        g = 1.0 if kind == "dirichlet" else 1.0 / math.sqrt(2.0)
        et, sg = math.sqrt(1.0 - g * g), SIGMA
        kb = 2.0 if kind == "absorbing_2beta" else 1.0
        sq = torch.sqrt(1.0 - kb * be * v)
        rho = et * (c2 * gu + al * gv) + g * c * sq * v
        rho = rho - et * (c2 * gue + al * gve) - g * c * torch.sqrt(1.0 - kb * be * vex) * vex
        return c2 * gu + al * gv - (et + sg * g) * rho, -(g - sg * et) / (c * sq) * rho

    def srct(self, t):
        return math.sin(16 * math.pi * t) * math.sin(math.pi * t) ** 2 if t < 1.0 else 0.0

    def rhs(self, U, V, t):
        N, nu, nv, h2 = self.N, self.nu, self.nv, self.th2
        P, D, w = self.P, self.D, self.w
        Pv, Dv = P[:, :nv], D[:, :nv]
        ein = torch.einsum
        back = lambda L, X, R: ein("ra,jkrs,sb->jkab", L, X, R)  # noqa: E731
        fwd = lambda L, X, R: ein("ra,jkab,sb->jkrs", L, X, R)  # noqa: E731
        uy, ux, vy, vx = fwd(D, U, P), fwd(P, U, D), fwd(Dv, V, Pv), fwd(Pv, V, Dv)
        F1, F2 = self.Cw * uy + self.Aw * vy, self.Cw * ux + self.Aw * vx
        R = -h2 * h2 * (back(Dv, F1, Pv) + back(Pv, F2, Dv))
        b = back(D, self.Cw * vy, P) + back(P, self.Cw * vx, D)
        th, tau, lu, lv = self.fl
        ct, st = (math.cos(self.om * t), math.sin(self.om * t)) if self.mms else (0.0, 0.0)
        for ax in (0, 1):
            # traces at the low and the high side, [j, k, i] along the face, 2/h times the derivatives
            ends = "jkab,a,ib->jki" if ax == 0 else "jkab,b,ia->jki"
            du = [h2 * ein(ends, U, self.E1[s], P) for s in (0, 1)]
            vv = [ein(ends, V, self.E[s, :nv], Pv) for s in (0, 1)]
            dv = [h2 * ein(ends, V, self.E1[s, :nv], Pv) for s in (0, 1)]
            c2, al, be = self.fc2[2 * ax:2 * ax + 2], self.fal[2 * ax:2 * ax + 2], self.fbe[2 * ax:2 * ax + 2]
            lo = lambda x: x[1:] if ax == 0 else x[:, 1:]  # noqa: E731      elements above a face: their low side
            hi = lambda x: x[:-1] if ax == 0 else x[:, :-1]  # noqa: E731
            c2m, c2p, am, ap = hi(c2[1]), lo(c2[0]), hi(al[1]), lo(al[0])
            dum, dup, dvm, dvp, sj = hi(du[1]), lo(du[0]), hi(dv[1]), lo(dv[0]), hi(vv[1]) - lo(vv[0])
            K = self.jc[ax] if self.jc is not None else 0.0
            J = c2m * dum - c2p * dup + am * dvm - ap * dvp + K
            G = (1 - th) * (c2m * dum + am * dvm) + th * (c2p * dup + ap * dvp)
            pen = 0.5 * (c2m + c2p) * lu + 0.5 * (am + ap) * lv
            wp, wm = th * sj - tau * J, -(1 - th) * sj - tau * J
            inner = ((pen * sj - G - (1 - th) * K, -ap * wp, c2p * wp), (G - pen * sj - th * K, am * wm, -c2m * wm))
            for s in (0, 1):
                edge = 0 if s == 0 else N - 1
                pick = (lambda x: x[edge]) if ax == 0 else (lambda x: x[:, edge])
                sgn = -1.0 if s == 0 else 1.0
                A, dvb = self.boundary(2 * ax + s, t, pick(c2[s]), pick(al[s]), pick(be[s]), pick(vv[s]),
                                       sgn * pick(du[s]), sgn * pick(dv[s]))
                slots = (A, sgn * pick(al[s]) * dvb, -sgn * pick(c2[s]) * dvb)
                full = [torch.cat([o.unsqueeze(ax), i] if s == 0 else [i, o.unsqueeze(ax)], ax)
                        for o, i in zip(slots, inner[s])]
                YA, YD, YF = (ein("jki,i,ib->jkb", f, w, Q) for f, Q in zip(full, (Pv, Pv, P)))
                lift = "a,jkb->jkab" if ax == 0 else "b,jka->jkab"
                R = R + h2 * ein(lift, self.E[s, :nv], YA) + h2 * h2 * ein(lift, self.E1[s, :nv], YD)
                b = b - ein(lift, self.E1[s], YF)
        if self.mms:
            o = self.om
            R = R - o * o * ct * self.pS - 2 * o ** 3 * st * ct * self.pB + (1 - ct) * self.pC + o * st * self.pD
        elif self.src:
            R = R + self.srct(t) * self.srcP
        else:
            R = R + self.pC
        first = torch.zeros(nu, nu, dtype=torch.float64, device=b.device)
        first[0, 0] = 1.0
        b = b + V[:, :, :1, :1] * first
        return self.solve_u(b), self.solve_v(V, R)

    def solve_u(self, b):
        N, nu = self.N, self.nu
        B = b.reshape(N * N, nu * nu)
        if self.case["coef"] in ("const", "cells"):     # A = c2 A1 away from the pinned constant mode
            X = torch.linalg.solve(self.A1, B.T).T
            s = (1.0 / self.c2q[:, :, 0, 0]).reshape(N * N, 1).expand(-1, nu * nu - 1)
            return (X * torch.cat([torch.ones_like(s[:, :1]), s], 1)).reshape(b.shape)
        Gx = torch.einsum("ra,sb->rsab", self.P, self.D).reshape(nu * nu, nu * nu)
        Gy = torch.einsum("ra,sb->rsab", self.D, self.P).reshape(nu * nu, nu * nu)
        out = []
        for C, r in zip(self.Cw.reshape(N * N, nu * nu, 1).split(8192), B.split(8192)):
            A = Gx.T @ (C * Gx) + Gy.T @ (C * Gy)
            A[:, 0, 0] += 1.0
            out.append(torch.linalg.solve(A, r))
        return torch.cat(out).reshape(b.shape)

    def solve_v(self, V, R):
        N, nv, qh = self.N, self.nv, self.qh
        vq = torch.einsum("ra,jkab,sb->jkrs", self.Ph, V, self.Ph)
        m = ((1.0 - 2.0 * self.beh * vq) * self.W).reshape(N * N, qh * qh, 1)
        out = [torch.linalg.solve(self.Phi.T @ (c * self.Phi), r)
               for c, r in zip(m.split(8192), R.reshape(N * N, nv * nv).split(8192))]
        return torch.cat(out).reshape(R.shape)

    def step(self, u, v, t, dt):
        k1, l1 = self.rhs(u, v, t)
        k2, l2 = self.rhs(u + 0.5 * dt * k1, v + 0.5 * dt * l1, t + 0.5 * dt)
        k3, l3 = self.rhs(u + 0.5 * dt * k2, v + 0.5 * dt * l2, t + 0.5 * dt)
        k4, l4 = self.rhs(u + dt * k3, v + dt * l3, t + dt)
        return u + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4), v + dt / 6 * (l1 + 2 * l2 + 2 * l3 + l4)

    def values(self, V):
        return torch.einsum("ra,jkab,sb->jkrs", self.P[:, :self.nv], V, self.P[:, :self.nv])

    def energy(self, u, v):
        P, D, h = self.P, self.D, 1.0 / self.N
        ux = self.th2 * torch.einsum("ra,jkab,sb->jkrs", P, u, D)
        uy = self.th2 * torch.einsum("ra,jkab,sb->jkrs", D, u, P)
        vh = self.values(v)
        Z = 0.5 * self.c2q * (ux * ux + uy * uy) + (0.5 - (2 / 3) * self.beq * vh) * vh * vh
        e = h * h / 4 * (Z * self.w[:, None] * self.w).sum()
        return float(e), float(vh.abs().max()), float((1 - 2 * self.beq * vh).min())


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = [exact(c, s) for c, s in _parts(case, seed)]
        return [u for u, _ in got] + [v for _, v in got]
    u, v = _state(case, seed)
    t, dt = _t0(seed), _dt(case, seed)
    M = _Dense(case, seed, grads=kind == "adjoint")
    if kind in ("rhs", "rhs_host"):
        k = M.rhs(u, v, t)
        return tuple(_flat(x) for x in k) if kind == "rhs" else tuple(_host(x) for x in k)
    if kind == "rk4":
        for _ in range(case["steps"]):
            u, v = M.step(u, v, t, dt)
            t += dt
        return _flat(u), _flat(v)
    if kind == "adjoint":
        lu, lv = (x / x.abs().max() for x in _state({**case, "state": "smooth"}, seed + 5))
        states, ts = [(u, v)], [t]
        with torch.no_grad():
            for _ in range(case["steps"] - 1):
                states.append(M.step(*states[-1], ts[-1], dt))
                ts.append(ts[-1] + dt)
        g = [0.0, 0.0, 0.0]
        for (a, b), t in zip(reversed(states), reversed(ts)):   # one step's graph at a time
            M = _Dense(case, seed, grads=True)
            a, b = a.detach().requires_grad_(True), b.detach().requires_grad_(True)
            a1, b1 = M.step(a, b, t, dt)
            lu, lv, *d = torch.autograd.grad((a1 * lu).sum() + (b1 * lv).sum(), (a, b, M.c2, M.al, M.be))
            g = [x + y for x, y in zip(g, d)]
        return tuple(_host(x) for x in (lu, lv, *g))
    N, nv = case["N"], M.nv
    row = lambda r: M.T(_basis(nv, np.array([r]))[0][0])  # noqa: E731
    at = [(_locate(y, N), _locate(x, N)) for x, y in RECEIVERS]
    j0, eta = _locate(SLICE_Y, N)
    recv, series, slices = [], [], []
    for it in range(1, case["steps"] + 1):
        u, v = M.step(u, v, t, dt)
        t += dt
        recv.append([float(row(a[1]) @ v[a[0], b[0]] @ row(b[1])) for a, b in at])
        if it % RECORD == 0 or it == case["steps"]:
            series.append(M.energy(u, v))
            slices.append(torch.einsum("a,kab,sb->ks", row(eta), v[j0], M.P[:, :nv]).reshape(-1).cpu().numpy())
    e = np.array(series)
    G = M.values(v).permute(0, 2, 1, 3).reshape(N * M.nu, N * M.nu)
    return dict(u=_host(u), v=_host(v), recv=np.array(recv), energy=e[:, 0], vmax=e[:, 1], ndmin=e[:, 2],
                slices=np.array(slices), snap=G.cpu().numpy())
