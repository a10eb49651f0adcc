"""Performance cases: what a program that uses ibpm_gpu has it do, through its
public Python entry points, from one step of a 64x64 grid to the two-cylinder
1024x1024 run.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges;
``prepare`` builds what a program holds before the call (the problem with its
Schur complement, a start state), ``run`` is one pass, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the same outputs from a plain
float64 torch restatement of the method (unit-source Schur complement
included), written independently of the library.

The start states are a few Gaussian vortices drawn from the seed around an
impulsively started body (the start of the repository's own benchmark) at 2 to
6 degrees of incidence; bodies sit a seeded 1e-3 ... 1e-2 h off the grid
lines, where the smoothed delta's rounded coefficients do not jump.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "ibpm.jl_b200", "python"))

import ibpm_gpu as G  # noqa: E402

# The transform lengths the library has (nx and ny), for draw().
LENGTHS = (64, 128, 192, 200, 256, 384, 400, 512)


def listed():
    return [
        # one advance per call with every field copied back, as a control or
        # coupling loop calls it: the smallest grid of the test suite
        dict(name="step_64", kind="advance", nx=64, ny=64, mg=3, bodies=1, Re=40.0, cfl=0.16, steps=1,
             precision="fp64"),
        # the reference's own cylinder benchmark: 200 cells (not a power of
        # two), three levels, 20 steps between looks at the state
        dict(name="cylinder_200", kind="advance", nx=200, ny=200, mg=3, bodies=1, Re=40.0, cfl=0.2, steps=20,
             precision="fp64"),
        # a single-level wide grid, FP32-refined: no nested levels at all
        dict(name="channel_256x128", kind="advance", nx=256, ny=128, mg=1, bodies=1, Re=100.0, cfl=0.2, steps=10,
             precision="fp32_refined"),
        # the pitching-plate benchmark on a moving grid (400x200, five levels):
        # the base flux changes every step
        dict(name="moving_grid_400x200", kind="moving_grid", nx=400, ny=200, mg=5, bodies=0, Re=100.0, cfl=0.05,
             steps=20, precision="fp64"),
        # the same plate moving through a fixed grid: the Schur complement is
        # rebuilt and inverted every step
        dict(name="moving_body_400x200", kind="moving_body", nx=400, ny=200, mg=5, bodies=0, Re=100.0, cfl=0.05,
             steps=4, precision="fp64"),
        # the headline workload: cylinder, 512x512 x 5 levels, in both precisions
        dict(name="cylinder_512", kind="advance", nx=512, ny=512, mg=5, bodies=1, Re=100.0, cfl=0.2, steps=40,
             precision="fp64"),
        dict(name="cylinder_512_refined", kind="advance", nx=512, ny=512, mg=5, bodies=1, Re=100.0, cfl=0.2,
             steps=10, precision="fp32_refined"),
        # the large two-body workload, 2512 force components
        dict(name="two_cylinders_1024", kind="advance", nx=1024, ny=1024, mg=5, bodies=2, Re=150.0, cfl=0.2,
             steps=20, precision="fp64"),
        # gradient of the mean force with respect to the start and the body
        # points: forward, recomputation and reverse sweep from a checkpoint
        dict(name="adjoint_256", kind="adjoint", nx=256, ny=256, mg=4, bodies=1, Re=100.0, cfl=0.2, steps=20,
             precision="fp64"),
        # one application of the linearised propagator, as a Krylov stability
        # run calls it: perturbation in, perturbation out
        dict(name="linearised_128", kind="linearised", nx=128, ny=128, mg=2, bodies=1, Re=40.0, cfl=0.2, steps=10,
             precision="fp64"),
        # a parameter sweep: members of several grids stepped together, each
        # member's forces and circulation read back
        dict(name="batch_16", kind="batch", nx=128, ny=384, mg=5, bodies=16, Re=100.0, cfl=0.2, steps=10,
             precision="fp32_refined"),
        # a new geometry: create a problem (its Schur complement and inverse),
        # read the inverse, release it, as a shape sweep or a
        # finite-difference check does
        dict(name="setup_200", kind="setup", nx=200, ny=200, mg=3, bodies=1, Re=40.0, cfl=0.2, steps=0,
             precision="fp64"),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["advance"] * 4 + ["moving_grid", "moving_body", "adjoint", "linearised", "setup"])
    small = kind in ("moving_body", "adjoint", "setup")
    while True:
        nx, ny = rng.choice(LENGTHS), rng.choice(LENGTHS)
        if ny <= nx <= 4 * ny and nx * ny <= (256 * 256 if small else 512 * 512):
            break
    mg = rng.randint(1, 5)
    steps = {"moving_body": rng.randint(1, 4), "adjoint": rng.randint(4, 16), "setup": 0}.get(
        kind, int(round(math.exp(rng.uniform(0.0, math.log(20))))))
    precision = rng.choice(["fp64", "fp32_refined"]) if kind in ("advance", "moving_grid") else "fp64"
    bodies = 0 if kind.startswith("moving") or rng.random() < 0.3 else 1
    return dict(kind=kind, nx=nx, ny=ny, mg=mg, bodies=bodies, Re=float(round(rng.uniform(40.0, 200.0), 1)),
                cfl=round(rng.uniform(0.05, 0.2), 3), steps=steps if precision == "fp64" else min(steps, 10),
                precision=precision)


# ---------------------------------------------------------------------------
# Problems and start states (host side)
# ---------------------------------------------------------------------------
def _grid(nx, ny, mg):
    """A domain of height 4 upstream-heavy in x, as the repository's grids."""
    h = 4.0 / ny
    return G.make_grid(h, (-0.25 * nx * h, 0.75 * nx * h, -2.0, 2.0), mg)


def _bodies(case, g, rng):
    dx, dy = (g.h * rng.uniform(1e-3, 1e-2, 2)).tolist()
    n = case["bodies"]
    if n == 0:     # flat plate with points h apart
        return [G.make_plate(1.0, 0.0, g.h, dx, dy, n=int(round(1.0 / g.h)) + 1)]
    r, m = 0.5, int(math.floor(math.pi / g.h / (1.0 if g.nx >= 200 else 2.0)))
    if n == 1:
        return [G.make_cylinder(r, g.h, dx, dy, n=m)]
    return [G.make_cylinder(r, g.h, dx, 0.75 + dy, n=m), G.make_cylinder(r, g.h, dx, -0.75 + dy, n=m)]


def _vorticity(g, rng, amp):
    """Γ (nΓ, mg) of four Gaussian vortices on the finest level."""
    X = np.arange(1, g.nx)[:, None] * g.h - g.offx
    Y = np.arange(1, g.ny)[None, :] * g.h - g.offy
    w = np.zeros((g.nx - 1, g.ny - 1))
    for _ in range(4):
        x0, y0, s, a = rng.uniform(0.5, 1.5), rng.uniform(-1.0, 1.0), rng.uniform(0.15, 0.3), rng.normal()
        w += amp * a * np.exp(-((X - x0) ** 2 + (Y - y0) ** 2) / s ** 2)
    out = np.zeros((g.nGamma, g.mg), order="F")
    out[:, 0] = (g.h * g.h * w).flatten(order="F")
    return out


def _motion(kind, rng):
    """A pitching motion about the leading edge, smooth in t."""
    w, a, p = rng.uniform(1.5, 2.5), rng.uniform(0.1, 0.2), rng.uniform(0.0, 1.0)
    th = lambda t: -a * math.sin(w * t + p)            # noqa: E731
    thd = lambda t: -a * w * math.cos(w * t + p)       # noqa: E731
    one, zero = (lambda t: 1.0), (lambda t: 0.0)
    if kind == "moving_grid":
        return G.MovingGrid(U=one, V=zero, theta=th, theta_dot=thd)
    hv = lambda t: 0.05 * math.sin(w * t)              # noqa: E731
    hvd = lambda t: 0.05 * w * math.cos(w * t)         # noqa: E731
    return G.MotionFunction(xc=(zero, hv, th), uc=(zero, hvd, thd))


def _inputs(case, seed):
    """The host-side description of a case: grid, bodies, dt, free stream,
    motion, start vorticity (from the seed alone)."""
    rng = np.random.default_rng([seed, 77])
    g = _grid(case["nx"], case["ny"], case["mg"])
    bodies = _bodies(case, g, rng)
    motion = _motion(case["kind"], rng) if case["kind"].startswith("moving") else None
    for b in bodies:
        b.motion = motion
    fs = (0.0, 0.0, 0.0) if case["kind"] == "moving_grid" else (1.0, 0.0, float(rng.uniform(0.03, 0.1)))
    return dict(g=g, bodies=bodies, dt=case["cfl"] * g.h, Re=case["Re"], fs=fs, motion=motion,
                gamma=_vorticity(g, rng, 0.5), base=_vorticity(g, rng, 1.0))


def _batch_specs(case, seed):
    rng = np.random.default_rng([seed, 78])
    specs, starts = [], []
    for i in range(case["bodies"]):
        n = (case["nx"], 192, 256, case["ny"])[i % 4]
        g = _grid(n, n, 3 + i % (case["mg"] - 2) if i >= 8 else case["mg"] - 1)
        one = dict(case, nx=n, ny=n, bodies=int(rng.integers(0, 2)))
        specs.append(dict(grid=g, bodies=_bodies(one, g, rng), dt=case["cfl"] * g.h,
                          Re=float(rng.uniform(40.0, 200.0)), precision=case["precision"],
                          freestream=(1.0, 0.0, float(rng.uniform(0.03, 0.1)))))
        starts.append(_vorticity(g, rng, 0.5))
    return specs, starts


def _start(prob, gamma):
    """A state consistent with Γ on the device and on the host: what a program
    has after building its start."""
    st = G.pinned_state(prob)
    st.Gamma[...] = gamma
    G.push_state(st, prob, fields=("Gamma",))
    G.vort2flux(st, prob)
    return st


def prepare(case, seed):
    if case["kind"] == "batch":
        specs, starts = _batch_specs(case, seed)
        batch = G.Batch(specs)
        sts = [_start(m, s) for m, s in zip(batch.members, starts)]
        return dict(case=case, batch=batch, sts=sts)
    c = _inputs(case, seed)
    if case["kind"] == "setup":
        return dict(case=case, c=c)
    prob = G.IBProblem(c["g"], c["bodies"], c["dt"], c["Re"], freestream=c["fs"], precision=case["precision"])
    s = dict(case=case, c=c, prob=prob, t=0.1)
    if case["kind"] == "linearised":
        base = _start(prob, c["base"])
        prob.set_base_state(base)
    s["st"] = _start(prob, c["gamma"])
    if case["kind"] in ("adjoint", "linearised"):
        s["start"], s["res"] = s["st"], G.pinned_state(prob)
    return s


def _fields(st, cd, cl):
    return dict(CD=cd, CL=cl, Gamma=st.Gamma, q=st.q, psi=st.psi, nonlin=st.nonlin[0], Fb=st.Fb)


def run(state):
    case = state["case"]
    n = case["steps"]
    if case["kind"] == "setup":
        c = state["c"]
        prob = G.IBProblem(c["g"], c["bodies"], c["dt"], c["Re"], freestream=c["fs"], precision=case["precision"])
        binv = prob.binv()
        prob.close()
        return binv
    if case["kind"] == "batch":
        forces = state["batch"].advance(n)
        for m, st in zip(state["batch"].members, state["sts"]):
            m._check(m.lib.ibpm_get_state(m.handle, G._ptr(st.Gamma), *[None] * 6))
        return [dict(CD=cd, CL=cl, Gamma=st.Gamma) for (cd, cl), st in zip(forces, state["sts"])]
    prob = state["prob"]
    if case["kind"] == "adjoint":
        G.push_state(state["start"], prob)
        r = G.adjoint_run(prob, n, k_checkpoint=max(1, n // 2), window=max(1, n // 2), w_cd=1.0, w_cl=0.5,
                          want_xb=True)
        return dict(J=np.array([r.J]), Gamma=r.grad_Gamma0, q=r.grad_q0, omega=r.grad_omega0,
                    alpha=np.array([r.grad_alpha]), xb=r.grad_xb)
    if case["kind"] == "linearised":
        G.push_state(state["start"], prob)
        cd, cl = G.advance(state["res"], prob, 0.0, nsteps=n)
        return _fields(state["res"], cd, cl)
    st = state["st"]
    ts = state["t"] + _dt(state) * np.arange(n)
    state["t"] += n * _dt(state)
    cd, cl = G.advance(st, prob, ts)
    return _fields(st, cd, cl)


def _dt(state):
    return state["c"]["dt"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(nx, ny, mg, nf):
    """One step: every operator reads its inputs and writes its outputs once
    (each 2-D transform one read and one write of a field), the Schur solve
    reads the inverse once; a transform costs 2.5 N log2 N per real line."""
    nG = (nx - 1) * (ny - 1)
    byt = 8.0 * nG * (34.5 * mg + 3.5) + 8.0 * nf * nf
    lines = 2.5 * nG * (math.log2(nx) + math.log2(ny))
    flops = (6.0 * mg + 2.0) * lines + 80.0 * nG * mg + 2.0 * nf * nf
    return byt, flops


def work(case):
    k, n = case["kind"], case["steps"]
    if k == "batch":
        specs, _ = _batch_specs(case, 1)
        w = [_step_work(s["grid"].nx, s["grid"].ny, s["grid"].mg, 2 * len(s["bodies"][0].xb)) for s in specs]
        back = sum(8.0 * s["grid"].nGamma * s["grid"].mg for s in specs)
        return dict(bytes=n * sum(a for a, _ in w) + back, flops=n * sum(b for _, b in w))
    c = _inputs(case, 1)
    g = c["g"]
    nf = 2 * sum(len(b.xb) for b in c["bodies"])
    byt, flops = _step_work(g.nx, g.ny, g.mg, nf)
    nG = float(g.nGamma)
    # one column of the Schur complement: A⁻¹ of one level, vort2flux of all
    col_b, col_f = 16.0 * nG * (2 + 2.5 * g.mg), 5.0 * nG * (math.log2(g.nx) + math.log2(g.ny)) * (1 + g.mg)
    inv_f = 2.0 * nf ** 3
    state = 8.0 * (3 * nG * g.mg + g.nq * g.mg)
    if k == "setup":
        return dict(bytes=nf * col_b + 16.0 * nf * nf, flops=nf * col_f + inv_f)
    if k == "moving_body":
        return dict(bytes=n * (byt + nf * col_b) + state, flops=n * (flops + nf * col_f + inv_f))
    if k == "adjoint":     # forward, recomputation and the transposed step
        return dict(bytes=3.5 * n * byt + 2 * state, flops=3.5 * n * flops)
    if k == "linearised":
        return dict(bytes=n * byt + 2 * state, flops=n * flops)
    return dict(bytes=n * byt + state, flops=n * flops)


# ---------------------------------------------------------------------------
# The same outputs in plain float64 torch
# ---------------------------------------------------------------------------
def _dst(x, dim):
    """DST-I along dim: Y_k = 2 Σ_j x_j sin(π (j+1)(k+1)/N), by the FFT of the
    odd extension."""
    n = x.shape[dim]
    z = torch.zeros_like(x.narrow(dim, 0, 1))
    f = torch.fft.rfft(torch.cat([z, x, z, -x.flip(dim)], dim), dim=dim)
    return -f.imag.narrow(dim, 1, n)


def _delta(r, h):
    """The smoothed delta of Yang et al. (2009) with 10-digit coefficients."""
    r = r.abs() / h
    r1 = r.clamp(0, 1)
    r2 = r.clamp(1, 2)
    r3 = r.clamp(2, 3)
    s3 = math.sqrt(3.0)

    def piece1(x):
        a, b = torch.asin(0.5 * s3 * (2 * x - 1)), torch.sqrt(1 - 12 * x ** 2 + 12 * x)
        return (4.166666667e-2 * x ** 4 + (-0.1388888889 + 3.472222222e-2 * b) * x ** 3
                + (-7.121664902e-2 - 5.208333333e-2 * b + 0.2405626122 * a) * x ** 2
                + (-.2405626122 * a - 0.3792313933 + 0.1012731481 * b) * x + 8.0187537413e-2 * a
                - 4.195601852e-2 * b + 0.6485698427)

    def piece2(x):
        a, b = torch.asin(0.5 * s3 * (2 * x - 3)), torch.sqrt(-23 + 36 * x - 12 * x ** 2)
        return (-6.250000000e-2 * x ** 4 + (0.4861111111 - 1.736111111e-2 * b) * x ** 3
                + (-1.143175026 + 7.812500000e-2 * b - 0.1202813061 * a) * x ** 2
                + (0.8751991178 + 0.3608439183 * a - 0.1548032407 * b) * x - 0.2806563809 * a
                + 8.22848104e-3 + 0.1150173611 * b)

    def piece3(x):
        a, b = torch.asin(0.5 * s3 * (2 * x - 5)), torch.sqrt(-71 - 12 * x ** 2 + 60 * x)
        return (2.083333333e-2 * x ** 4 + (3.472222222e-3 * b - 0.2638888889) * x ** 3
                + (1.214391675 - 2.604166667e-2 * b + 2.405626122e-2 * a) * x ** 2
                + (-0.1202813061 * a - 2.449273192 + 7.262731481e-2 * b) * x + 0.1523563211 * a
                + 1.843201677 - 7.306134259e-2 * b)

    out = torch.where(r <= 1, piece1(r1), torch.where(r <= 2, piece2(r2), piece3(r3)))
    return torch.where(r <= 3, out, torch.zeros_like(out))


class _Plain:
    """The method on arrays of rows along y: Γ-like (mg, ny-1, nx-1), fluxes
    (mg, ny, nx+1) and (mg, ny+1, nx), float64, differentiable."""

    def __init__(self, c, dev):
        g, self.dev = c["g"], dev
        self.nx, self.ny, self.mg, self.h = g.nx, g.ny, g.mg, g.h
        self.offx, self.offy = g.offx, g.offy
        self.dt, self.Re, self.motion = c["dt"], c["Re"], c["motion"]
        self.npts = [len(b.xb) for b in c["bodies"]]
        self.x0 = torch.tensor(np.concatenate([b.xb for b in c["bodies"]]), device=dev)
        k = torch.arange(1, max(g.nx, g.ny), dtype=torch.float64, device=dev)
        ex = 4 * torch.sin(0.5 * math.pi * k[:g.nx - 1] / g.nx) ** 2
        ey = 4 * torch.sin(0.5 * math.pi * k[:g.ny - 1] / g.ny) ** 2
        self.lam = ey[:, None] + ex[None, :]
        self.hc = [g.h * 2.0 ** l for l in range(g.mg)]
        self.base = None
        self.ub = None
        U, V, a = c["fs"]
        self.set_alpha(U, V, torch.tensor(a, dtype=torch.float64, device=dev))
        self.place(self.x0)

    def set_alpha(self, U, V, a):
        self.q0x = [(U * torch.cos(a) - V * torch.sin(a)) * hc for hc in self.hc]
        self.q0y = [(U * torch.sin(a) + V * torch.cos(a)) * hc for hc in self.hc]

    # Poisson-type solves
    def lap_inv(self, f):
        w = _dst(_dst(f, -1), -2) / self.lam
        return _dst(_dst(w, -1), -2) / (4.0 * self.nx * self.ny)

    def a_inv(self, f, lev):
        M = 1 + self.lam * (self.dt / (2 * self.Re * self.hc[lev] ** 2))
        w = _dst(_dst(f, -1), -2) / M
        return _dst(_dst(w, -1), -2) / (4.0 * self.nx * self.ny)

    # edge values of a level sampled from the next coarser one, indexed by vertex
    def get_bc(self, r):
        nx, ny = self.nx, self.ny

        def fill(s):
            mid = 0.5 * (s[..., 1:] + s[..., :-1])
            out = torch.stack([s[..., :-1], mid], -1).flatten(-2)
            return torch.cat([out, s[..., -1:]], -1)
        xs, ys = slice(nx // 4 - 1, 3 * nx // 4), slice(ny // 4 - 1, 3 * ny // 4)
        return (fill(r[..., ny // 4 - 1, xs]), fill(r[..., 3 * ny // 4 - 1, xs]),
                fill(r[..., ys, nx // 4 - 1]), fill(r[..., ys, 3 * nx // 4 - 1]))

    def zero_bc(self, r):
        z = lambda n: torch.zeros(r.shape[:-2] + (n,), dtype=r.dtype, device=r.device)  # noqa: E731
        return z(self.nx + 1), z(self.nx + 1), z(self.ny + 1), z(self.ny + 1)

    def apply_bc(self, r, bc, fac):
        b, t, le, ri = bc
        r = r.clone()
        r[..., 0, :] += fac * b[..., 1:-1]
        r[..., -1, :] += fac * t[..., 1:-1]
        r[..., :, 0] += fac * le[..., 1:-1]
        r[..., :, -1] += fac * ri[..., 1:-1]
        return r

    def coarsify(self, levels):
        nx, ny = self.nx, self.ny
        out = [levels[0]]
        for lev in range(1, len(levels)):
            f = out[-1]
            row = f[..., 1:-1:2, :] + 0.5 * (f[..., 0:-2:2, :] + f[..., 2::2, :])
            cen = row[..., :, 1:-1:2] + 0.5 * (row[..., :, 0:-2:2] + row[..., :, 2::2])
            lv = levels[lev].clone()
            lv[..., ny // 4:3 * ny // 4 - 1, nx // 4:3 * nx // 4 - 1] = cen
            out.append(lv)
        return out

    def curl(self, p, bc):
        b, t, le, ri = bc
        nx = self.nx
        # the bottom edge value of an x-flux is taken one vertex to the left
        # of the top one's (the reference's index)
        lo = torch.cat([b[..., 0:nx - 1].unsqueeze(-2), p], -2)
        hi = torch.cat([p, t[..., 1:-1].unsqueeze(-2)], -2)
        qx = torch.cat([(le[..., 1:] - le[..., :-1]).unsqueeze(-1), hi - lo,
                        (ri[..., 1:] - ri[..., :-1]).unsqueeze(-1)], -1)
        w = torch.cat([le[..., 1:-1].unsqueeze(-1), p], -1)
        e = torch.cat([p, ri[..., 1:-1].unsqueeze(-1)], -1)
        qy = torch.cat([(b[..., :-1] - b[..., 1:]).unsqueeze(-2), w - e, (t[..., :-1] - t[..., 1:]).unsqueeze(-2)], -2)
        return qx, qy

    def rot(self, qx, qy):
        return ((qx[..., :-1, 1:-1] - qx[..., 1:, 1:-1]) + (qy[..., 1:-1, 1:] - qy[..., 1:-1, :-1]))

    def vort2flux(self, levels, want=None):
        levels = self.coarsify(levels)
        psi, q, bc = [None] * self.mg, [None] * self.mg, None
        for lev in range(self.mg - 1, -1, -1):
            f = levels[lev]
            if lev < self.mg - 1:
                bc = self.get_bc(psi[lev + 1])
                f = self.apply_bc(f, bc, 1.0)
            else:
                bc = self.zero_bc(f)
            psi[lev] = self.lap_inv(f)
            if want is None or lev < want:
                q[lev] = self.curl(psi[lev], bc)
        return levels, psi, q

    # coupling: windows of 13x13 flux points around each body point
    def place(self, xb, built=None):
        h, s = self.h, torch.arange(-6, 7, device=self.dev)
        xd = xb.detach()
        bx = torch.floor((xd[:, 0] + self.offx) / h).long()
        by = torch.floor((xd[:, 1] + self.offy) / h).long()
        I, J = bx[:, None] + s - 1, by[:, None] + s - 1
        x, y = h * I.double() - self.offx, h * J.double() - self.offy
        X, Y = xb[:, 0:1], xb[:, 1:2]
        self.wx = _delta(y + h / 2 - Y, h)[:, :, None] * _delta(x - X, h)[:, None, :]
        self.wy = _delta(y - Y, h)[:, :, None] * _delta(x + h / 2 - X, h)[:, None, :]
        self.I, self.J = I, J

    def E(self, qx, qy):
        J, I = self.J[:, :, None], self.I[:, None, :]
        fx = (qx[..., J, I] * self.wx).sum((-1, -2))
        fy = (qy[..., J, I] * self.wy).sum((-1, -2))
        return torch.cat([fx, fy], -1)

    def EtC(self, f):
        nb, lead = self.I.shape[0], f.shape[:-1]
        nx, ny = self.nx, self.ny
        J, I = self.J[:, :, None], self.I[:, None, :]
        ax = (J * (nx + 1) + I).reshape(-1)
        ay = (J * nx + I).reshape(-1)
        fx = (f[..., :nb, None, None] * self.wx).reshape(lead + (-1,))
        fy = (f[..., nb:, None, None] * self.wy).reshape(lead + (-1,))
        qx = torch.zeros(lead + (ny * (nx + 1),), dtype=f.dtype, device=f.device).index_add(-1, ax, fx)
        qy = torch.zeros(lead + ((ny + 1) * nx,), dtype=f.dtype, device=f.device).index_add(-1, ay, fy)
        return self.rot(qx.reshape(lead + (ny, nx + 1)), qy.reshape(lead + (ny + 1, nx)))

    def B_times(self, Z):
        g0 = self.a_inv(self.EtC(Z), 0)
        levels = [g0] + [torch.zeros_like(g0) for _ in range(self.mg - 1)]
        _, _, q = self.vort2flux(levels, want=1)
        return self.E(*q[0])

    def build(self):
        nf = 2 * self.I.shape[0]
        eye = torch.eye(nf, dtype=torch.float64, device=self.dev)
        per = max(1, int(3e7 / (self.nx * self.ny * self.mg)))
        with torch.no_grad():
            self.B = torch.cat([self.B_times(eye[k:k + per]) for k in range(0, nf, per)]).T.contiguous()
            self.Binv = torch.linalg.inv(self.B)

    def solve_B(self, F):
        if not torch.is_grad_enabled():
            return self.Binv @ F
        # x = B⁻¹F with the derivative of B carried by one application of B:
        # dx = B⁻¹(dF − dB x)
        x = (self.Binv @ F).detach()
        return x + self.Binv @ (F - self.B_times(x))

    def move(self, t):
        m = self.motion
        x, y, th = (float(f(t)) for f in m.xc)
        xd, yd, thd = (float(f(t)) for f in m.uc)
        c, s = math.cos(th), math.sin(th)
        X, Y = self.x0[:, 0], self.x0[:, 1]
        self.ub = torch.cat([xd - thd * (s * X + c * Y), yd + thd * (c * X - s * Y)])
        self.place(torch.stack([x + c * X - s * Y, y + s * X + c * Y], 1))
        self.build()

    def index(self, n):
        return torch.arange(n, dtype=torch.float64, device=self.dev)

    def grid_flux(self, t):
        """Base flux of a moving grid at t, per level: (ny, 1) and (1, nx)."""
        m = self.motion
        a, Om = -m.theta(t), -m.theta_dot(t)
        Ux = m.U(t) * math.cos(a) - m.V(t) * math.sin(a)
        Uy = m.U(t) * math.sin(a) + m.V(t) * math.cos(a)
        for l, hc in enumerate(self.hc):
            y = (self.index(self.ny) + 0.5 - self.ny / 2) * hc + self.ny / 2 * self.h - self.offy
            x = (self.index(self.nx) + 0.5 - self.nx / 2) * hc + self.nx / 2 * self.h - self.offx
            self.q0x[l] = (-hc * Om * y + hc * Ux)[:, None]
            self.q0y[l] = (hc * Om * x + hc * Uy)[None, :]

    def product(self, Qx, Qy, Gm, bc):
        b, t, le, ri = bc
        v = torch.cat([b[1:-1][None], Gm, t[1:-1][None]], 0)
        hz = torch.cat([le[1:-1][:, None], Gm, ri[1:-1][:, None]], 1)
        fx = Qy[1:] * v[1:] + Qy[:-1] * v[:-1]
        fy = -(Qx[:, 1:] * hz[:, 1:] + Qx[:, :-1] * hz[:, :-1])
        return ((fx[:-1] - fx[1:]) + (fy[:, 1:] - fy[:, :-1]))

    def face_sums(self, qx, qy, lev, with_base):
        ux = qx + self.q0x[lev] if with_base else qx
        uy = qy + self.q0y[lev] if with_base else qy
        return ux[1:] + ux[:-1], uy[:, 1:] + uy[:, :-1]

    def step(self, Gm, q, Nprev, t):
        if self.motion is not None:
            if hasattr(self.motion, "theta_dot"):
                self.grid_flux(t)
            else:
                self.move(t)
        N, S = [], []
        for l in range(self.mg):
            hc = self.hc[l]
            bc = self.get_bc(Gm[l + 1]) if l + 1 < self.mg else self.zero_bc(Gm[l])
            b4 = tuple(0.25 * v for v in bc)
            if self.base is None:
                n = self.product(*self.face_sums(*q[l], l, True), Gm[l], b4)
            else:
                GB, QB = self.base
                n = (self.product(*self.face_sums(*q[l], l, False), GB[l], b4)
                     + self.product(*QB[l], Gm[l], b4))
            n = n / (4 * hc ** 2)
            c = self.dt / (2 * self.Re * hc ** 2)
            g = torch.nn.functional.pad(Gm[l], (1, 1, 1, 1))
            lap = g[1:-1, 2:] + g[1:-1, :-2] + g[2:, 1:-1] + g[:-2, 1:-1] - 4 * Gm[l]
            r = Gm[l] + c * lap + 1.5 * self.dt * n - 0.5 * self.dt * Nprev[l]
            r = self.apply_bc(r, bc, 0.25 * self.dt / (self.Re * hc ** 2))
            N.append(n)
            S.append(self.a_inv(r, l))
        S, _, qs = self.vort2flux(S, want=1)
        zero = self.base is not None
        F = self.E(qs[0][0] + (0.0 if zero else self.q0x[0]), qs[0][1] + (0.0 if zero else self.q0y[0]))
        if self.ub is not None:
            F = F - self.ub * self.h
        Fb = self.solve_B(F)
        S = list(S)
        S[0] = S[0] - self.a_inv(self.EtC(Fb), 0)
        Gn, psi, qn = self.vort2flux(S)
        return Gn, qn, N, psi, Fb

    def forces(self, Fb):
        nb, cd, cl, p = self.I.shape[0], [], [], 0
        for n in self.npts:
            cd.append(2 * self.h / self.dt * Fb[p:p + n].sum())
            cl.append(2 * self.h / self.dt * Fb[nb + p:nb + p + n].sum())
            p += n
        return torch.stack(cd), torch.stack(cl)

    def levels(self, ref):
        t = torch.tensor(np.ascontiguousarray(ref.T), device=self.dev)
        return [t[l].reshape(self.ny - 1, self.nx - 1) for l in range(self.mg)]

    def column(self, levels):
        return torch.stack([v.reshape(-1) for v in levels], 1)

    def flux_column(self, q):
        return torch.stack([torch.cat([a.reshape(-1), b.reshape(-1)]) for a, b in q], 1)


def exact(case, seed):
    if case["kind"] == "batch" or case["nx"] * case["ny"] * case["mg"] > 3e6:
        return None     # a batch is its members; the 1024x1024 Schur complement takes minutes
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    c = _inputs(case, seed)
    p = _Plain(c, dev)
    n = case["steps"]
    if case["kind"] != "moving_body":
        p.build()
    if case["kind"] == "setup":
        return p.Binv
    zero = [torch.zeros(p.ny - 1, p.nx - 1, dtype=torch.float64, device=dev) for _ in range(p.mg)]
    if case["kind"] == "adjoint":
        return _exact_gradient(p, c, case, zero)
    with torch.no_grad():
        if case["kind"] == "linearised":
            GB, _, qB = p.vort2flux(p.levels(c["base"]))
            QB = [p.face_sums(*qB[l], l, True) for l in range(p.mg)]
            p.base = (GB, QB)
        Gm, psi, q = p.vort2flux(p.levels(c["gamma"]))
        N, cds, cls, Fb = zero, [], [], None
        for k in range(n):
            Gm, q, N, psi, Fb = p.step(Gm, q, N, 0.1 + k * c["dt"])
            cd, cl = p.forces(Fb)
            cds.append(cd)
            cls.append(cl)
        return dict(CD=torch.stack(cds), CL=torch.stack(cls), Gamma=p.column(Gm), q=p.flux_column(q),
                    psi=p.column(psi), nonlin=p.column(N), Fb=Fb[:, None])


def _exact_gradient(p, c, case, zero):
    """The gradient of the windowed mean of CD + CL/2 by automatic
    differentiation of the plain step."""
    n, w = case["steps"], max(1, case["steps"] // 2)
    dev = p.dev
    with torch.no_grad():
        G0, _, q0 = p.vort2flux(p.levels(c["gamma"]))
    with torch.enable_grad():
        al = torch.tensor(c["fs"][2], dtype=torch.float64, device=dev, requires_grad=True)
        p.set_alpha(c["fs"][0], c["fs"][1], al)
        xb = p.x0.clone().requires_grad_(True)
        p.place(xb)
        G0 = [v.clone().requires_grad_(True) for v in G0]
        q0 = [(a.clone().requires_grad_(True), b.clone().requires_grad_(True)) for a, b in q0]
        Gm, q, N, J = G0, q0, zero, 0.0
        for k in range(n):
            Gm, q, N, _, Fb = p.step(Gm, q, N, 0.0)
            if k >= n - w:
                cd, cl = p.forces(Fb)
                J = J + (cd + 0.5 * cl).sum() / w
        flat = [v for v in G0] + [v for ab in q0 for v in ab] + [al, xb]
        gr = torch.autograd.grad(J, flat)
        gG, gq = gr[:p.mg], [(gr[p.mg + 2 * l], gr[p.mg + 2 * l + 1]) for l in range(p.mg)]
        # a start built from a finest-level vorticity ω: Γ₀ = coarsify([h²ω, 0 …]), q₀ = curl ψ(Γ₀)
        om = zero[0].clone().requires_grad_(True)
        lv, _, qv = p.vort2flux([p.h ** 2 * om] + zero[1:])
        s = sum((a * b).sum() for a, b in zip(lv, gG))
        s = s + sum((a * x).sum() + (b * y).sum() for (a, b), (x, y) in zip(qv, gq))
        gw, = torch.autograd.grad(s, om)
    return dict(J=J.detach().reshape(1), Gamma=p.column(gG), q=p.flux_column(gq), omega=gw.reshape(-1),
                alpha=gr[-2].reshape(1), xb=gr[-1])
