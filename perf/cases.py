"""What the solver is used for, as calls a program makes: the sizes and options
below are those of the package's own generators, tests and benchmark.

A pass is a number of outer iterations (or a thermal solve) through the public
Python binding, the fields back on the host included; iteration counts are
fixed (no stop test) because the 1e-6 stop of a whole solve is one dip of a
wandering residual and moves with the last bit of every sum.

kinds
  start    a solve from the zero state: the first outer iterations, whose
           pressure PCG runs to its cap (more than half of a solve's time)
  restart  a solve continued from stored fields: the late regime, Jacobi sweeps
           and about one PCG iteration per outer iteration
  steps    the drop-in's use: one outer iteration per call and the planes the
           outer loop samples after it
  batch    designs of uneven size advanced together on groups of CTAs
  thermal  the 3-D conjugate-heat-transfer solve of a design
"""
import math

import numpy as np
import torch

from coldplate_solver_b200 import batch, cps, geometry, thermal


def listed():
    return [
        # the 2-D straight channel, FOU, uvAlpha 0.7, PCG capped at 20: the smallest grid
        # anyone solves in earnest, bound by the latency of each phase
        dict(name="channel 200x100 start", kind="start", geometry="channel", M=100, N=200, mixed=False, iters=60),
        # the same channel driven step by step by a program that owns the outer loop
        dict(name="channel 200x100 steps", kind="steps", geometry="channel", M=100, N=200, mixed=False, iters=12),
        # the 2.5-D channel network, SOU, PCG capped at 20
        dict(name="network 500x250 start", kind="start", geometry="network", M=250, N=500, mixed=False, iters=60),
        # a small served request picked up again from its stored fields
        dict(name="density 256x128 restart", kind="restart", geometry="density", M=128, N=256, mixed=False, iters=300),
        # density-field designs (SOU, Brinkman, 2.5-D, PCG capped at 200), mixed precision as served
        dict(name="density 512x256 mixed", kind="start", geometry="density", M=256, N=512, mixed=True, iters=12),
        # the benchmark's design: its first iterations, and its late ones in both precisions
        dict(name="density 1000x500 start", kind="start", geometry="density", M=500, N=1000, mixed=False, iters=12),
        dict(name="density 1000x500 restart", kind="restart", geometry="density", M=500, N=1000, mixed=False, iters=300),
        dict(name="density 1000x500 mixed", kind="restart", geometry="density", M=500, N=1000, mixed=True, iters=300),
        # the largest grid of the served stream
        dict(name="density 2048x1024 start", kind="start", geometry="density", M=1024, N=2048, mixed=False, iters=6),
        # designs of a mix, log-uniform sizes, advanced together
        dict(name="mix of 8 start", kind="batch", geometry="density", M=0, N=512, mixed=False, iters=12, designs=8,
             mix=1),
        # the heat-transfer solve, 2 base-plate layers under 7 channel layers
        dict(name="thermal 250x125x9", kind="thermal", geometry="density", M=125, N=250, mixed=False, iters=0),
        dict(name="thermal 1000x500x9", kind="thermal", geometry="density", M=500, N=1000, mixed=False, iters=0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["start", "start", "start", "restart", "restart", "steps", "batch", "thermal"])
    geo = rng.choice(["density", "density", "channel", "network"]) if kind in ("start", "restart", "steps") else "density"
    n = {"start": log(96, 1600), "restart": log(128, 1000), "steps": log(96, 400), "batch": log(256, 700),
         "thermal": log(100, 1000)}[kind]
    m = max(40, int(n * rng.uniform(0.4, 0.6)))
    c = dict(kind=kind, geometry=geo, M=0 if kind == "batch" else m, N=n, mixed=kind != "thermal" and rng.random() < 0.3,
             iters={"start": rng.randint(4, 12), "restart": rng.randint(60, 300), "steps": rng.randint(4, 20),
                    "batch": rng.randint(4, 12), "thermal": 0}[kind])
    if kind == "batch":
        c["designs"], c["mix"] = rng.randint(3, 8), rng.randrange(1 << 20)
    return c


# ---------------------------------------------------------------- inputs
def _density_gamma(M, N, seed):
    """Blurred (sigma 8 cells), tanh-projected noise, open at both ends."""
    rng = np.random.default_rng(seed)
    f = np.fft.rfft2(rng.random((M, N)))
    ky, kx = np.fft.fftfreq(M)[:, None], np.fft.rfftfreq(N)[None, :]
    s = np.fft.irfft2(f * np.exp(-2.0 * (math.pi * 8.0) ** 2 * (ky * ky + kx * kx)), s=(M, N))
    s = (s - s.min()) / (s.max() - s.min())
    t = math.tanh(4.0)
    g = np.clip((t + np.tanh(8.0 * (s - 0.5))) / (2.0 * t), 0.0, 1.0)
    w = min(8, N // 4)
    g[1:M - 2, :w] = 1.0
    g[1:M - 2, N - w:] = 1.0
    return g


def _design(geo, M, N, seed):
    rng = np.random.default_rng([seed, 1])
    if geo == "channel":
        return geometry.straight_channel(M=M, N=N, U=float(rng.uniform(0.08, 0.12)))
    if geo == "network":
        return geometry.channel_network(M=M, N=N, seed=seed, U=float(rng.uniform(0.15, 0.25)))
    alpha, gamma = geometry.alpha_ramp_q(_density_gamma(M, N, seed))
    return geometry.Design(M=M, N=N, hx=10e-6, hy=10e-6, inletVelocity=float(rng.uniform(0.08, 0.2)), gamma=gamma,
                           alpha=alpha, convectionScheme=1, enableTwoPointFiveD=True, enableConvectionScaling=True,
                           Ht_channel=300e-6, twoPointFiveDSinkMultiplier=1.0, uvAlpha=0.3, pAlpha=0.1,
                           maxPressureIter=200)


def _batch_designs(case, seed):
    """Log-uniform widths from a quarter of N up to N; which ones is the mix."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for k in range(case["designs"]):
        n = int(round(math.exp(rng.uniform(math.log(case["N"] / 4), math.log(case["N"])))))
        out.append(_design("density", max(20, n // 2), n, seed + 1000 * (k + 1)))
    return out


def _thermal_case(case, seed):
    """A density field and a mass-conserving flow through it: every column
    carries the same flow, spread over its cells by their permeability."""
    M, N, h = case["M"], case["N"], 10e-6
    g = _density_gamma(M, N, seed)
    w = g + 0.02
    u = 0.1 * M * w / w.sum(axis=0)
    psi = np.vstack([np.zeros(N), np.cumsum(u, axis=0)])  # at the rows' edges
    v = -np.gradient(0.5 * (psi[1:] + psi[:-1]), axis=1)
    q = float(np.random.default_rng([seed, 3]).uniform(0.5e6, 1.5e6))
    return thermal.ThermalCase(gamma=g, u=u, v=v, dx=h, dy=h, q=q, H_t=300e-6)


def _warm_iters(case):
    """Outer iterations after which the PCG has left its cap (density designs
    of these sizes do so within about N)."""
    return max(250, case["N"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "thermal":
        return dict(case=case, solver=thermal.ThermalSolver(_thermal_case(case, seed)))
    precision = cps.CPS_MIXED if case["mixed"] else cps.CPS_FP64
    if kind == "batch":
        solvers = [cps.Solver(d, precision=precision) for d in _batch_designs(case, seed)]
        return dict(case=case, solvers=solvers, mode=batch.default_mode())
    solver = cps.Solver(_design(case["geometry"], case["M"], case["N"], seed), precision=precision)
    state = dict(case=case, solver=solver)
    if kind == "restart":
        solver.solve(_warm_iters(case), eps=0.0)
        f = solver.download()
        state["fields"] = {k: f[k] for k in ("u", "v", "p")}
    return state


# ---------------------------------------------------------------- the calls
def _outputs(hist, fields):
    hist = np.asarray(hist)
    return dict(residuals=np.ascontiguousarray(hist[:, :5]), counts=hist[:, 5:8].astype(np.int64),
                u=fields["u"], v=fields["v"], p=fields["p"], uStar=fields["uStar"], vStar=fields["vStar"],
                dE=fields["dE"], dN=fields["dN"])


def run(state):
    case = state["case"]
    kind, iters = case["kind"], case["iters"]
    if kind == "thermal":
        state["solver"].solve()
        return dict(T=state["solver"].temperature())
    if kind == "batch":
        for s in state["solvers"]:
            s.reset_fields()
        res, _ = cps.batch_solve(state["solvers"], iters, eps=0.0, **state["mode"])
        out = dict(last=np.array([r["last"][:5] for r in res]),
                   counts=np.array([[r["n_done"], *r["last"][5:8]] for r in res], dtype=np.int64))
        for k, s in enumerate(state["solvers"]):
            f = s.download()
            out["fields%d" % k] = [f["u"], f["v"], f["p"]]
        return out
    s = state["solver"]
    if kind == "restart":
        s.upload_fields(**state["fields"])
        return _outputs(s.solve(iters, eps=0.0), s.download())
    s.reset_fields()
    if kind == "start":
        return _outputs(s.solve(iters, eps=0.0), s.download())
    hist, planes = [], []
    xs = _planes(s.design)
    for _ in range(iters):
        d = s.step()
        hist.append([d[k] for k in ("residU", "residV", "residMass", "residMassDof", "err", "pIters", "uSweeps",
                                    "vSweeps")])
        planes.append([s.sample_plane(x) for x in xs])
    out = _outputs(hist, s.download())
    out["planes"] = np.array(planes)
    return out


def _planes(d):
    """The core's ends and the domain's ends."""
    L = d.N * d.hx
    return (0.2 * L, 0.8 * L, 0.0, L)


def _cells(case):
    if case["kind"] == "batch":  # the mean of the log-uniform widths' squares
        n = case["N"]
        return int(case["designs"] * 0.5 * n * n * (1 - 1 / 16.0) / (2 * math.log(4)))
    return case["M"] * case["N"]


def work(case):
    """Inputs once and outputs once; the operations of the method's formulas
    (assembly, sweeps, PCG, correction; the heat solve at 60 iterations of two
    V-cycles and two products)."""
    n, kind = _cells(case), case["kind"]
    if kind == "thermal":
        return {"bytes": 8.0 * n * (4 + 9), "flops": 60.0 * 9 * n * 2 * (4 * 1.33 * 16 + 16 + 8)}
    cg = 2 if kind == "restart" else (200 if case["geometry"] == "density" else 20)
    per = 330 + 5 * 11 + 21 * cg
    planes = 1 if kind == "batch" else 2
    return {"bytes": 8.0 * n * (3 * (kind == "restart") + 2 + 3 * planes + (2 if planes == 2 else 0)),
            "flops": float(per) * n * case["iters"]}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _pad(a):
    return torch.nn.functional.pad(a, (2, 2, 2, 2))


class _Flow:
    """The outer iteration on whole arrays."""

    def __init__(self, d):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.d, M, N = d, d.M, d.N
        f = dict(dtype=torch.float64, device=self.dev)
        self.u, self.v, self.p = torch.zeros(M + 1, N, **f), torch.zeros(M, N + 1, **f), torch.zeros(M + 1, N + 1, **f)
        self.alpha, self.gamma = torch.tensor(d.alpha, **f), torch.tensor(d.gamma, **f)
        self.mv = 3.0 * max(abs(d.inletVelocity), 0.1)

    def clamp(self, x):
        return x.clamp(-self.mv, self.mv)

    def momentum(self, is_u):
        """Solves one component; returns (x, d coefficient, sweeps) over its unknowns."""
        d, M, N = self.d, self.d.M, self.d.N
        i1, j1 = (M - 1, N - 2) if is_u else (M - 2, N - 1)
        I, J = torch.arange(1, i1 + 1, device=self.dev)[:, None], torch.arange(1, j1 + 1, device=self.dev)[None, :]

        def at(pad, di, dj):
            return pad[3 + di:3 + di + i1, 3 + dj:3 + dj + j1]

        U, V, X = _pad(self.u), _pad(self.v), _pad(self.u if is_u else self.v)
        A, Pp = _pad(self.alpha), _pad(self.p)
        if is_u:
            drag = 0.5 * (at(A, -1, -1) + at(A, -1, 0))
            ue, uw = 0.5 * (at(U, 0, 0) + at(U, 0, 1)), 0.5 * (at(U, 0, -1) + at(U, 0, 0))
            vn, vs = 0.5 * (at(V, 0, 0) + at(V, 0, 1)), 0.5 * (at(V, -1, 0) + at(V, -1, 1))
            force = (at(Pp, 0, 0) - at(Pp, 0, 1)) * d.hy
        else:
            drag = 0.5 * (at(A, -1, -1) + at(A, 0, -1))
            ue, uw = 0.5 * (at(U, 0, 0) + at(U, 1, 0)), 0.5 * (at(U, 0, -1) + at(U, 1, -1))
            vn, vs = 0.5 * (at(V, 0, 0) + at(V, 1, 0)), 0.5 * (at(V, -1, 0) + at(V, 0, 0))
            force = (at(Pp, 0, 0) - at(Pp, 1, 0)) * d.hx
        scale = 6.0 / 7.0 if d.enableConvectionScaling else 1.0
        Fe, Fw = scale * d.rho * d.hy * self.clamp(ue), scale * d.rho * d.hy * self.clamp(uw)
        Fn, Fs = scale * d.rho * d.hx * self.clamp(vn), scale * d.rho * d.hx * self.clamp(vs)
        De, Dn = d.eta * d.hy / d.hx, d.eta * d.hx / d.hy
        aE, aW = De + (-Fe).clamp(min=0), De + Fw.clamp(min=0)
        aN, aS = Dn + (-Fn).clamp(min=0), Dn + Fs.clamp(min=0)
        sink = 0.0
        if d.enableTwoPointFiveD and d.Ht_channel > 0:
            sink = d.twoPointFiveDSinkMultiplier * 5.0 * d.eta / (2.0 * d.Ht_channel ** 2)
        vol = d.hx * d.hy
        aP0 = (aE + aW + aN + aS + (Fe - Fw + Fn - Fs) + sink * vol + drag * vol).clamp(min=1e-10)
        aP = aP0 / d.uvAlpha
        x = at(X, 0, 0).clone()
        b = force + (1.0 - d.uvAlpha) / d.uvAlpha * aP0 * x
        if d.convectionScheme == 1:
            c, e, w, n, s = at(X, 0, 0), at(X, 0, 1), at(X, 0, -1), at(X, 1, 0), at(X, -1, 0)
            jm, im = (N - 1, M) if is_u else (N, M - 1)  # last index of the component's plane

            def up(F, ok, near, far, sign):  # second-order upwind minus first-order, times the flux
                return sign * torch.where(ok, F * (0.5 * near - 0.5 * far), torch.zeros_like(F))

            b = b + torch.where(Fe >= 0, up(Fe, (J >= 2) & (I > 0), c, w, -1),
                                up(Fe, (J + 2 <= jm) & (I > 0), e, at(X, 0, 2), -1))
            b = b + torch.where(Fw >= 0, up(Fw, (J >= 2) & (I > 0), w, at(X, 0, -2), 1),
                                up(Fw, (J + 1 <= jm) & (I > 0), c, e, 1))
            b = b + torch.where(Fn >= 0, up(Fn, (I >= 1) & (J > 0), c, s, -1),
                                up(Fn, (I + 2 <= im) & (J > 0), n, at(X, 2, 0), -1))
            b = b + torch.where(Fs >= 0, up(Fs, (I >= 2) & (J > 0), s, at(X, -2, 0), 1),
                                up(Fs, (I + 1 <= im) & (J > 0), c, n, 1))
        for a, (di, dj), inside in ((aE, (0, 1), J + 1 <= j1), (aW, (0, -1), J > 1), (aN, (1, 0), I + 1 <= i1),
                                    (aS, (-1, 0), I > 1)):
            b = b + torch.where(inside.expand_as(a), torch.zeros_like(a), a * at(X, di, dj))
        tol, sweeps = d.momentumTol ** 2 * i1 * j1, 0
        while sweeps < d.maxMomentumIter:
            q = torch.nn.functional.pad(x, (1, 1, 1, 1))
            r = b - (aP * x - aE * q[1:-1, 2:] - aW * q[1:-1, :-2] - aN * q[2:, 1:-1] - aS * q[:-2, 1:-1])
            x = x + r / aP
            sweeps += 1
            if float((r * r).sum()) < tol:
                break
        return self.clamp(x), (d.hy if is_u else d.hx) / aP0, sweeps

    def step(self):
        d, M, N = self.d, self.d.M, self.d.N
        xu, eU, ku = self.momentum(True)
        xv, eV, kv = self.momentum(False)
        us, vs = torch.zeros_like(self.u), torch.zeros_like(self.v)
        dE, dN = torch.zeros_like(self.u), torch.zeros_like(self.v)
        inlet = (self.gamma[:M - 1, 0] > 0.5).to(torch.float64) * d.inletVelocity
        us[1:M, 1:N - 1], vs[1:M - 1, 1:N] = xu, xv
        dE[1:M, 1:N - 1], dN[1:M - 1, 1:N] = eU, eV
        ru, rv = float((us - self.u)[1:M, 1:N - 1].abs().max()), float((vs - self.v)[1:M - 1, 1:N].abs().max())
        us[1:M, N - 1], us[1:M, 0], vs[1:M - 1, N] = us[1:M, N - 2], inlet, vs[1:M - 1, N - 1]
        b = d.rho * d.hy * (us[1:M, :N - 1] - us[1:M, 1:N]) + d.rho * d.hx * (vs[:M - 1, 1:N] - vs[1:M, 1:N])
        rm, rd = float(b.abs().max()), float(b[:, :-1].abs().max())
        x, its = self.pcg(b[:, :-1], d.rho * d.hy * dE[1:M, 0:N - 1], d.rho * d.hx * dN[0:M, 1:N - 1])
        pc = torch.zeros_like(self.p)
        pc[1:M, 1:N - 1] = x
        p = self.p
        p[1:M, 1:N] += d.pAlpha * pc[1:M, 1:N]
        p[0, 1:N], p[M, 1:N], p[1:M, 0], p[1:M, N] = p[1, 1:N], p[M - 1, 1:N], p[1:M, 1], 0.0
        self.u, self.v = us.clone(), vs.clone()
        self.u[1:M, 1:N - 1] = self.clamp(xu + self.clamp(eU * (pc[1:M, 1:N - 1] - pc[1:M, 2:N])))
        self.v[1:M - 1, 1:N] = self.clamp(xv + self.clamp(eV * (pc[1:M - 1, 1:N] - pc[2:M, 1:N])))
        self.u[1:M, N - 1], self.v[1:M - 1, N] = self.u[1:M, N - 2], self.v[1:M - 1, N - 1]
        self.star = dict(uStar=us, vStar=vs, dE=dE, dN=dN)
        return [ru, rv, rm, rd, max(ru, rv, rm), its, ku, kv]

    def pcg(self, b, ce, cn):
        """ce: east-face conductances of columns 0..N-2, cn: north-face ones of rows 0..M-1 (zero at the walls)."""
        d = self.d
        W, E, S, Nn = ce[:, :-1], ce[:, 1:], cn[:-1], cn[1:]
        diag = E + W + Nn + S
        diag = torch.where(diag < 1e-20, torch.ones_like(diag), diag)
        x, r = torch.zeros_like(b), b.clone()
        z = r / diag
        p, rz = z.clone(), (r * z).sum()
        for it in range(d.maxPressureIter):
            q = torch.nn.functional.pad(p, (1, 1, 1, 1))
            Ap = diag * p - W * q[1:-1, :-2] - E * q[1:-1, 2:] - S * q[:-2, 1:-1] - Nn * q[2:, 1:-1]
            pAp = (p * Ap).sum()
            if abs(float(pAp)) < 1e-20:
                return x, it
            a = rz / pAp
            x += a * p
            r -= a * Ap
            if float((r * r).sum()) ** 0.5 < d.pTol:
                return x, it
            z = r / diag
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x, d.maxPressureIter

    def plane(self, xp):
        d, M, N = self.d, self.d.M, self.d.N
        x = min(max(xp, 0.5 * d.hx), (N - 0.5) * d.hx)
        c = max(0, min(int(math.floor(x / d.hx - 0.5)), N - 2))
        t = max(0.0, min(1.0, (x - (c + 0.5) * d.hx) / d.hx))
        open_ = (self.gamma[:M - 1, c] >= 1 - 1e-6) & (self.gamma[:M - 1, c + 1] >= 1 - 1e-6)
        st = (1 - t) * self.p[1:M, c + 1] + t * self.p[1:M, min(c + 2, N)]
        un = (1 - t) * self.u[1:M, c] + t * self.u[1:M, c + 1]
        vv = (1 - t) * self.v[:, c] + t * self.v[:, c + 1]
        vt = 0.5 * (vv[:M - 1] + vv[1:M])
        dyn = 0.5 * d.rho * (un * un + vt * vt)
        st, dyn, flux = st[open_], dyn[open_], (d.rho * un * d.hy).abs()[open_]
        area, fl = float(open_.sum()) * d.hy, float(flux.sum())
        s, y = (float(st.sum()) * d.hy / area, float(dyn.sum()) * d.hy / area) if area > 0 else (0.0, 0.0)
        tot = float(((st + dyn) * flux).sum()) / fl if fl > 0 else s + y
        return [area, fl, s, y, tot, float(area > 0)]


def _heat_system(c):
    """The seven coefficient planes (W E S N B T diagonal) and the source."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f = dict(dtype=torch.float64, device=dev)
    g, u, v = (torch.tensor(x, **f) for x in (c.gamma, c.u, c.v))
    nz = c.nz_solid + c.nz_fluid
    gam = g.clamp(0, 1)
    k = torch.full((nz, c.Ny, c.Nx), c.k_s, **f)
    k[c.nz_solid:] = c.k_f + (c.k_s - c.k_f) * (1 - gam) / (1 + c.qk * gam)
    z = (torch.arange(c.nz_fluid, **f) + 0.5) / c.nz_fluid
    po = torch.cat([torch.zeros(c.nz_solid, **f), 4 * z * (1 - z)])[:, None, None]
    fluid = torch.zeros(k.shape, dtype=torch.bool, device=dev)
    fluid[c.nz_solid:] = g > 0.01
    u3, v3 = u * po, v * po
    dz = torch.tensor([c.H_b / c.nz_solid] * c.nz_solid + [c.H_t / c.nz_fluid] * c.nz_fluid, **f)[:, None, None]
    rc, Ax, Ay, Az = c.rho * c.Cp, c.dy * dz, c.dx * dz, c.dx * c.dy
    W, E, S, N, B, T = (torch.zeros_like(k) for _ in range(6))
    diag, b = torch.zeros_like(k), torch.zeros_like(k)

    def harm(x, y):
        return 2 * x * y / (x + y + 1e-30)

    Dx, Dy = harm(k[:, :, 1:], k[:, :, :-1]) * Ax / c.dx, harm(k[:, 1:], k[:, :-1]) * Ay / c.dy
    Fx = torch.where(fluid[:, :, 1:] & fluid[:, :, :-1], rc * 0.5 * (u3[:, :, 1:] + u3[:, :, :-1]) * Ax, 0.0)
    Fy = torch.where(fluid[:, 1:] & fluid[:, :-1], rc * 0.5 * (v3[:, 1:] + v3[:, :-1]) * Ay, 0.0)
    W[:, :, 1:], E[:, :, :-1] = -Dx - Fx.clamp(min=0), -Dx - (-Fx).clamp(min=0)
    S[:, 1:], N[:, :-1] = -Dy - Fy.clamp(min=0), -Dy - (-Fy).clamp(min=0)
    diag[:, :, 1:] += Dx + (-Fx).clamp(min=0)
    diag[:, :, :-1] += Dx + Fx.clamp(min=0)
    diag[:, 1:] += Dy + (-Fy).clamp(min=0)
    diag[:, :-1] += Dy + Fy.clamp(min=0)
    Din, Fin = 2 * k[:, :, 0] * Ax[:, :, 0] / c.dx, rc * u3[:, :, 0] * Ax[:, :, 0]
    inl = fluid[:, :, 0]
    diag[:, :, 0] += torch.where(inl, Din + (-Fin).clamp(min=0), 0.0)
    b[:, :, 0] += torch.where(inl, (Din + Fin.clamp(min=0)) * c.T_inlet, 0.0)
    diag[:, :, -1] += torch.where(fluid[:, :, -1], (rc * u3[:, :, -1] * Ax[:, :, 0]).clamp(min=0), 0.0)
    diag[:, -1] += torch.where(fluid[:, -1], (rc * v3[:, -1] * Ay[:, :, 0]).clamp(min=0), 0.0)
    zP, zN = dz[:-1], dz[1:]
    Dz = (zP + zN) / (zP / k[:-1] + zN / k[1:]) * Az / (0.5 * (zP + zN))
    B[1:], T[:-1] = -Dz, -Dz
    diag[1:] += Dz
    diag[:-1] += Dz
    b[0] += c.q * Az
    return W, E, S, N, B, T, diag + 1e-12, b


def _heat_exact(c):
    """BiCGStab, line-preconditioned in z, to the rounding of 64 bits."""
    W, E, S, N, B, T, D, b = _heat_system(c)
    nz = D.shape[0]

    def mul(x):
        q = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
        return (D * x + W * q[1:-1, 1:-1, :-2] + E * q[1:-1, 1:-1, 2:] + S * q[1:-1, :-2, 1:-1]
                + N * q[1:-1, 2:, 1:-1] + B * q[:-2, 1:-1, 1:-1] + T * q[2:, 1:-1, 1:-1])

    m = [D[0]]
    for k in range(1, nz):
        m.append(D[k] - B[k] * T[k - 1] / m[k - 1])

    def line(r):
        y = [r[0]]
        for k in range(1, nz):
            y.append(r[k] - B[k] / m[k - 1] * y[k - 1])
        x = [y[-1] / m[-1]]
        for k in range(nz - 2, -1, -1):
            x.append((y[k] - T[k] * x[-1]) / m[k])
        return torch.stack(x[::-1])

    x = torch.full_like(b, c.T_inlet)
    nb, best, keep = b.norm(), math.inf, x
    for _ in range(4):  # restarted, so that the recurrence's residual is the true one
        r = b - mul(x)
        h, rho, p = r.clone(), (r * r).sum(), r.clone()
        for it in range(3000):
            ph = line(p)
            v = mul(ph)
            a = rho / (h * v).sum()
            s = r - a * v
            sh = line(s)
            t = mul(sh)
            w = (t * s).sum() / (t * t).sum()
            x = x + a * ph + w * sh
            r = s - w * t
            if it % 50 == 49 and float(r.norm() / nb) < 1e-14:
                break
            new = (h * r).sum()
            p = r + new / rho * a / w * (p - w * v)
            rho = new
        true = float((b - mul(x)).norm() / nb)
        if true < best:
            best, keep = true, x
        if not math.isfinite(true) or true < 1e-13:
            break
        x = keep.clone()
    return keep if best < 1e-11 else None


def exact(case, seed):
    kind = case["kind"]
    if kind == "thermal":
        if case["M"] * case["N"] > 50000:  # thousands of iterations of the plain method
            return None
        T = _heat_exact(_thermal_case(case, seed))
        return None if T is None else dict(T=T.cpu().numpy())
    if kind == "batch":
        flows, last, counts = [_Flow(d) for d in _batch_designs(case, seed)], [], []
        for f in flows:
            h = [f.step() for _ in range(case["iters"])][-1]
            last.append(h[:5])
            counts.append([case["iters"], *h[5:8]])
        out = dict(last=np.array(last), counts=np.array(counts, dtype=np.int64))
        for k, f in enumerate(flows):
            out["fields%d" % k] = [f.u.cpu().numpy(), f.v.cpu().numpy(), f.p.cpu().numpy()]
        return out
    if kind == "restart" and case["N"] > 300:  # hundreds of iterations to get there
        return None
    f = _Flow(_design(case["geometry"], case["M"], case["N"], seed))
    for _ in range(_warm_iters(case) if kind == "restart" else 0):
        f.step()
    hist, planes = [], []
    for _ in range(case["iters"]):
        hist.append(f.step())
        if kind == "steps":
            planes.append([f.plane(x) for x in _planes(f.d)])
    fields = dict(u=f.u, v=f.v, p=f.p, **f.star)
    out = _outputs(hist, {k: t.cpu().numpy() for k, t in fields.items()})
    if kind == "steps":
        out["planes"] = np.array(planes)
    return out
