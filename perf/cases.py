"""The work that is timed: what programs have this library do, over its range of sizes.

Each case is one pass through the public entry points (``Simulation``, its ``Solver``, ``BatchSolver``, the autograd
energy, the headless colormaps) as a program calls them in a loop.  ``listed`` names the cases, ``draw`` gives more of the
same ranges, ``prepare`` builds what such a program holds before the call (inputs, handle, workspace), ``run`` is the pass,
``exact`` computes the same results in 64 bits with plain torch, ``work`` counts the bytes and operations of a pass.

Inputs are solitons with noise (N(0, 1e-3)) and a vacuum ring: skyrmion lattices, hedgehogs, vortices at positions drawn
from the seed, at the lattice spacings of the parity configurations (chiral magnet h = 1/32, baby Skyrme 0.1, Abelian
Higgs 0.05, s+id 0.085).
"""
import math

import numpy as np
import torch

from soliton_solver_b200.autograd import coupling_gradients, energy
from soliton_solver_b200.core.batch import BatchSolver
from soliton_solver_b200.core.colormaps import render_jet_density_to_rgba, render_magnetization_to_rgba
from soliton_solver_b200.core.simulation import Simulation
from soliton_solver_b200.theories import load_theory

DEVICE = "cuda"
NF = {"chiral": 4, "baby": 3, "higgs": 4, "sid": 6}
TITLE = {"chiral": "Chiral magnet", "baby": "Baby Skyrme", "higgs": "Abelian Higgs", "sid": "s+id superconductor"}
SPACING = {"chiral": 1.0 / 32.0, "baby": 0.1, "higgs": 0.05, "sid": 0.085}
HALO = 2
# chiral magnet: physical constants (Heusler DMI, demag on, 0.2 T) and the reduced couplings they give
MAGNET = dict(J=40e-12, K=0.8e6, D=4e-3, M=580e3, B=0.2, mu0=1.25663706127e-6)
# s+id superconductor: free-energy coefficients
SID = dict(alpha1=-1.0, alpha2=-1.24503, beta1=1.0, beta2=1.4959, beta3=4.02498, beta4=1.006245, Q=1.0, kappa=0.673274,
           gamma1=1.0, gamma2=0.877868, gamma12=0.534484)
# floating-point operations of one gradient evaluation per site (jets of every component plus the theory's point)
GRADIENT_FLOPS = {"chiral": 150, "baby": 230, "higgs": 210, "sid": 420}
ENERGY_FLOPS = {"chiral": 50, "baby": 50, "higgs": 50, "sid": 120}


def listed():
    return [
        # one interactive step with its energy and err on the host, smallest parity lattice: call latency
        dict(name="step_baby_128_fp64", kind="step", theory="baby", prec="fp64", X=128, Y=128),
        # the same call on the default 256 x 256 lattice of the chiral magnet: a viewer's or a script's step loop
        dict(name="step_chiral_256", kind="step", theory="chiral", prec="fp32", X=256, Y=256),
        # a stretch of a relaxation of one anti-skyrmion, trajectories on the host: latency of a step
        dict(name="relax_chiral_320", kind="relax", theory="chiral", prec="fp32", X=320, Y=320, steps=100),
        # steps between two looks at a lattice whose rows are no multiple of 16 bytes
        dict(name="advance_baby_500x333", kind="advance", theory="baby", prec="fp32", X=500, Y=333, steps=40),
        # the heaviest theory (six components)
        dict(name="advance_sid_512", kind="advance", theory="sid", prec="fp32", X=512, Y=512, steps=20),
        # double-precision relaxation of four vortices (coupling studies)
        dict(name="relax_higgs_1024_fp64", kind="relax", theory="higgs", prec="fp64", X=1024, Y=1024, steps=10),
        # a large lattice of the Skyrme term's theory
        dict(name="advance_baby_2048", kind="advance", theory="baby", prec="fp32", X=2048, Y=2048, steps=10),
        # the largest: 64 anti-skyrmions, variants chosen by the tuner as a long run does
        dict(name="relax_chiral_4096", kind="relax", theory="chiral", prec="fp32", X=4096, Y=4096, steps=10, tuned=True),
        # a parameter sweep of many small lattices advanced together, replayed as one graph
        dict(name="sweep_baby_28", kind="sweep", theory="baby", prec="fp32", count=28, small=64, large=512, steps=20),
        # the numbers of a finished relaxation: energy, charges, energy density, coupling derivatives
        dict(name="observe_chiral_2048", kind="observe", theory="chiral", prec="fp32", X=2048, Y=2048),
        # the energy as a differentiable term: forward and backward
        dict(name="grad_higgs_1500x1000", kind="grad", theory="higgs", prec="fp32", X=1500, Y=1000),
        # one frame of a headless animation: steps, charge density, two images
        dict(name="frame_chiral_1280x720", kind="frame", theory="chiral", prec="fp32", X=1280, Y=720, steps=4),
    ]


def draw(rng):
    """One more case: kinds as listed, extents log-uniform over 48 .. 2048 (three in ten odd), steps so that a pass costs
    no more than the largest listed one."""
    kind = rng.choice(["step", "relax", "relax", "advance", "advance", "sweep", "observe", "grad", "frame"])

    def extent():
        n = int(round(math.exp(rng.uniform(math.log(48), math.log(2048)))))
        return n | 1 if rng.random() < 0.3 else max(48, n // 4 * 4)

    theory = {"frame": "chiral", "sweep": "baby"}.get(kind) or rng.choice(["chiral", "baby", "higgs", "sid"])
    prec = "fp32" if kind in ("advance", "sweep", "frame") or rng.random() < 0.5 else "fp64"
    # step and relax in FP32 are the chiral magnet's; the other theories' FP32 lattices are advanced between two looks
    if kind in ("step", "relax") and theory != "chiral":
        prec = "fp64"
    if kind == "sweep":
        return dict(kind=kind, theory=theory, prec=prec, count=rng.randint(4, 28), small=rng.choice([48, 64, 96]),
                    large=rng.choice([128, 192, 256, 384]), steps=rng.randint(5, 30))
    c = dict(kind=kind, theory=theory, prec=prec, X=extent(), Y=extent())
    if kind in ("relax", "advance"):
        c["steps"] = max(3, min(rng.randint(20, 100), int(1.2e7 / (c["X"] * c["Y"]))))
    if kind == "frame":
        c["steps"] = rng.randint(1, 6)
    return c


# --------------------------------------------------------------------------- inputs
def _sid_vacuum():
    s = SID
    theta = math.pi / 2 if s["beta4"] >= 0 else 0.0
    b3t = s["beta3"] + 2.0 * math.cos(2.0 * theta) * s["beta4"]
    den = b3t * b3t - 4.0 * s["beta1"] * s["beta2"]
    n1 = 2.0 * s["beta2"] * s["alpha1"] - b3t * s["alpha2"]
    n2 = 2.0 * s["beta1"] * s["alpha2"] - b3t * s["alpha1"]
    return (math.sqrt(n1 / den) if n1 / den > 0 else 0.0, math.sqrt(n2 / den) if n2 / den > 0 else 0.0, theta)


def _field(theory, X, Y, seed, dtype):
    """Initial field (nf, X, Y): solitons at seeded positions, noise, vacuum ring."""
    h = SPACING[theory]
    g = torch.Generator(device=DEVICE)
    g.manual_seed(1000003 * (seed + 1) + 8191 * X + Y)
    pos = np.random.default_rng([seed, X, Y])
    x = (torch.arange(X, device=DEVICE, dtype=torch.float64) * h)[:, None]
    y = (torch.arange(Y, device=DEVICE, dtype=torch.float64) * h)[None, :]
    Lx, Ly = (X - 1) * h, (Y - 1) * h
    noise = lambda k: 1e-3 * torch.randn((k, X, Y), device=DEVICE, dtype=torch.float64, generator=g)  # noqa: E731
    if theory in ("chiral", "baby"):
        # hedgehogs f = pi exp(-r/R) composed through their stereographic coordinates
        step, R = (16.0, 1.0) if theory == "chiral" else (26.0, 1.5)
        nx, ny = max(1, round(Lx / step)), max(1, round(Ly / step))
        wr = torch.zeros((X, Y), device=DEVICE, dtype=torch.float64)
        wi = torch.zeros_like(wr)
        for i in range(nx):
            for j in range(ny):
                dx = x - (i + 0.5 + 0.25 * (pos.random() - 0.5)) * Lx / nx
                dy = y - (j + 0.5 + 0.25 * (pos.random() - 0.5)) * Ly / ny
                r = torch.sqrt(dx * dx + dy * dy).clamp_(min=1e-12)
                t = torch.tan(0.5 * math.pi * torch.exp(-r / R)) / r
                if theory == "chiral":  # anti-skyrmion
                    wr -= t * dy
                    wi -= t * dx
                else:
                    wr += t * dx
                    wi += t * dy
        q = wr * wr + wi * wi
        m = torch.stack([2 * wr / (1 + q), 2 * wi / (1 + q), (1 - q) / (1 + q)]) + noise(3)
        m /= torch.sqrt((m * m).sum(0, keepdim=True))
        for a, v in enumerate((0.0, 0.0, 1.0)):
            m[a, :HALO] = v
            m[a, -HALO:] = v
            m[a, :, :HALO] = v
            m[a, :, -HALO:] = v
        F = torch.cat([m, torch.zeros((1, X, Y), device=DEVICE, dtype=torch.float64)]) if theory == "chiral" else m
    else:
        n = 4 if theory == "higgs" else 2
        re = torch.ones((X, Y), device=DEVICE, dtype=torch.float64)
        im = torch.zeros_like(re)
        for _ in range(n):
            dx = x - (0.25 + 0.5 * pos.random()) * Lx
            dy = y - (0.25 + 0.5 * pos.random()) * Ly
            r = torch.sqrt(dx * dx + dy * dy).clamp_(min=1e-12)
            a = torch.tanh(r) / r
            re, im = a * (re * dx - im * dy), a * (re * dy + im * dx)
        z = torch.zeros_like(re)
        if theory == "higgs":
            F = torch.stack([z, z, re, im])
        else:
            u1, u2, th = _sid_vacuum()
            c, s = math.cos(th), math.sin(th)
            F = torch.stack([z, z, u1 * re, u1 * im, u2 * (c * re + s * im), u2 * (c * im - s * re)])
        F = F + noise(F.shape[0])
    return F.to(dtype)


def _params(theory, X, Y):
    h = SPACING[theory]
    th = load_theory(TITLE[theory])
    kw = dict(xlen=X, ylen=Y, xsize=(X - 1) * h, ysize=(Y - 1) * h, lsx=h, lsy=h)
    if theory == "chiral":
        kw.update(MAGNET, dmi_term="Heusler", demag=True, unit_magnetization=True)
    elif theory == "baby":
        kw.update(kappa=1.0, mpi=1.0, time_step=0.01, unit_magnetization=True)
    elif theory == "higgs":
        kw.update(q=1.0, u1=1.0, vortex_number=1.0, Lambda=1.0)
    else:
        kw.update(SID)
    return th, th.params.default_params(**kw)


def _dtype(prec):
    return torch.float32 if prec == "fp32" else torch.float64


def _sweep_sizes(case):
    """Extents of the lattices: powers of two from `small` up to `large`, cycled."""
    sizes, s = [], int(case["small"])
    while s <= case["large"]:
        sizes.append(s)
        s *= 2
    return [sizes[i % len(sizes)] for i in range(case["count"])]


def prepare(case, seed):
    theory, prec = case["theory"], case["prec"]
    if case["kind"] == "sweep":
        plist = []
        th = None
        for i, n in enumerate(_sweep_sizes(case)):
            th, p = _params(theory, n, n)
            plist.append(p.with_(kappa=_sweep_kappa(i)))
        b = BatchSolver(th, plist, prec)
        for i, n in enumerate(_sweep_sizes(case)):
            b.load(i, _field(theory, n, n, seed + 101 * i, _dtype(prec)))
        b.capture(int(case["steps"]))
        return dict(case=case, batch=b)
    th, p = _params(theory, case["X"], case["Y"])
    sim = Simulation(p, th, precision=prec)
    sim.load_field(_field(theory, case["X"], case["Y"], seed, _dtype(prec)))
    if case.get("tuned"):
        sim.solver.autotune()
    state = dict(case=case, sim=sim, E=1e300)
    if case["kind"] == "grad":
        state["leaf"] = sim.Field.clone().requires_grad_(True)
    if case["kind"] == "frame":
        state["images"] = [torch.zeros((case["Y"], case["X"], 4), dtype=torch.uint8, device=DEVICE) for _ in range(2)]
    return state


def _sweep_kappa(i):
    return 0.5 + 0.05 * (i % 16)


# --------------------------------------------------------------------------- the pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sweep":
        b = state["batch"]
        b.replay()
        return list(b.fields) + list(b.velocities)
    sim = state["sim"]
    if kind == "step":
        state["E"], err = sim.step(state["E"])
        return dict(field=sim.Field, velocity=sim.Velocity, energy=state["E"], err=err)
    if kind == "relax":
        E, err = sim.relax(int(case["steps"]))
        return dict(field=sim.Field, velocity=sim.Velocity, energy=E, err=err)
    if kind == "advance":
        sim.solver.step_async(int(case["steps"]))
        return dict(field=sim.Field, velocity=sim.Velocity)
    if kind == "observe":
        obs = sim.observables()
        sim.compute_energy_density()
        return dict(obs=obs, density=sim.en, couplings=coupling_gradients(sim))
    if kind == "grad":
        leaf = state["leaf"]
        leaf.grad = None
        E = energy(leaf, sim.solver)
        E.backward()
        return dict(energy=E, grad=leaf.grad)
    # frame
    sim.solver.step_async(int(case["steps"]))
    sim.compute_skyrmion_density()
    X, Y = case["X"], case["Y"]
    jet, mag = state["images"]
    render_jet_density_to_rgba[None, None](jet, sim.en, X, Y, -1e-4, 1e-4)
    render_magnetization_to_rgba[None, None](mag, sim.Field, X, Y, sim.p_i_h)
    return dict(field=sim.Field, velocity=sim.Velocity, density=sim.en, jet=jet, magnetization=mag)


# --------------------------------------------------------------------------- work of a pass
def work(case):
    w = 4 if case["prec"] == "fp32" else 8
    t = case["theory"]
    if case["kind"] == "sweep":
        sites = float(sum(n * n for n in _sweep_sizes(case)))
    else:
        sites = float(case["X"] * case["Y"])
    field = NF[t] * w * sites
    if case["kind"] == "observe":
        # five reductions' worth of arithmetic over the field, read once; the energy density written
        return dict(bytes=field + 8 * sites, flops=6.0 * ENERGY_FLOPS[t] * sites)
    if case["kind"] == "grad":
        return dict(bytes=2 * field, flops=(GRADIENT_FLOPS[t] + ENERGY_FLOPS[t]) * sites)
    # a step reads and writes the field and the velocity; four gradients and one energy per step
    n = float(case.get("steps", 1))
    out = dict(bytes=4 * field * n, flops=(4 * GRADIENT_FLOPS[t] + ENERGY_FLOPS[t]) * sites * n)
    if case["kind"] == "frame":
        out["bytes"] += (3 * w + 8 + 8) * sites
        out["flops"] += 100.0 * sites
    return out


# --------------------------------------------------------------------------- the same in 64 bits
class _Exact:
    """The theories' energy, gradient and flow of an (nf, X, Y) field in float64 torch: 4th-order central stencils, zero
    within HALO of the edge (the mixed derivative from the main diagonal, one row and column further in at the low side)."""

    def __init__(self, theory, X, Y, kappa=1.0):
        self.t, self.X, self.Y, self.h, self.kappa = theory, X, Y, SPACING[theory], kappa
        self.dA = self.h * self.h
        self.dt = 0.01 if theory == "baby" else 0.5 * self.h
        x = torch.arange(X, device=DEVICE)[:, None]
        y = torch.arange(Y, device=DEVICE)[None, :]
        self.mx = ((x >= HALO) & (x <= X - HALO - 1)).double()
        self.my = ((y >= HALO) & (y <= Y - HALO - 1)).double()
        self.mxy = ((x > HALO) & (x < X - HALO) & (y > HALO) & (y < Y - HALO)).double()
        c = MAGNET
        self.cK = c["K"] * c["J"] / c["D"] ** 2
        self.ch = c["M"] * c["B"] * c["J"] / c["D"] ** 2
        self.cmu = c["mu0"] * c["M"] ** 2 * c["J"] / c["D"] ** 2

    def jet(self, f, second=True):
        p = torch.nn.functional.pad(f[None, None], (2, 2, 2, 2))[0, 0]
        X, Y, h = self.X, self.Y, self.h

        def s(i, j):
            return p[2 + i:2 + i + X, 2 + j:2 + j + Y]

        def first(a, b):
            return (2.0 / 3.0 * (s(a, b) - s(-a, -b)) - (s(2 * a, 2 * b) - s(-2 * a, -2 * b)) / 12.0) / h

        def raw(a, b):
            return (4.0 / 3.0 * (s(a, b) - 2 * f + s(-a, -b)) - (s(2 * a, 2 * b) - 2 * f + s(-2 * a, -2 * b)) / 12.0)

        out = [first(1, 0) * self.mx, first(0, 1) * self.my]
        if second:
            xx, yy = raw(1, 0) / h ** 2, raw(0, 1) / h ** 2
            out += [xx * self.mx, yy * self.my]
            out.append((raw(1, 1) / (2 * self.dA) - 0.5 * (xx + yy)) * self.mxy)
        return out

    def energy_density(self, F):
        d = [self.jet(f, False) for f in F]
        if self.t == "chiral":
            e = sum(0.5 * (d[a][0] ** 2 + d[a][1] ** 2) for a in range(3))
            m = F[:3]
            # Heusler DMI: D00 = 1, D11 = -1
            e = e + m[1] * d[2][0] - m[2] * d[1][0] + m[0] * d[2][1] - m[2] * d[0][1]
            e = e - F[3] * (d[0][0] + d[1][1]) - (d[3][0] ** 2 + d[3][1] ** 2) / (2 * self.cmu)
            e = e + self.ch * (1 - m[2]) + self.cK * (1 - m[2] ** 2)
        elif self.t == "baby":
            c = torch.linalg.cross(torch.stack([v[0] for v in d]), torch.stack([v[1] for v in d]), dim=0)
            e = 0.5 * sum(v[0] ** 2 + v[1] ** 2 for v in d) + 0.5 * self.kappa ** 2 * (c * c).sum(0) + 1 - F[2]
        elif self.t == "higgs":
            q = F[2] ** 2 + F[3] ** 2
            e = 0.5 * (d[2][0] ** 2 + d[2][1] ** 2 + d[3][0] ** 2 + d[3][1] ** 2)
            for i in range(2):
                e = e + F[i] * (F[2] * d[3][i] - F[3] * d[2][i])
            e = e + 0.5 * (F[0] ** 2 + F[1] ** 2) * q + (1 - q) ** 2 / 8.0 + 0.5 * (d[1][0] - d[0][1]) ** 2
        else:
            s = SID
            u1, u2, th = _sid_vacuum()

            def pot(ar, ai, br, bi):
                a, b = ar * ar + ai * ai, br * br + bi * bi
                # Re(conj(p1)^2 p2^2) = (ar br + ai bi)^2 - (ar bi - ai br)^2
                cross = (ar * br + ai * bi) ** 2 - (ar * bi - ai * br) ** 2
                return (s["alpha1"] * a + s["alpha2"] * b + s["beta1"] * a * a + s["beta2"] * b * b + s["beta3"] * a * b
                        + 2 * s["beta4"] * cross)

            e = pot(F[2], F[3], F[4], F[5]) + 0.5 * s["kappa"] ** 2 * (d[1][0] - d[0][1]) ** 2
            for i in range(2):
                g = self._gamma(i)
                Dr, Di = self._cov(F, d, i)
                for a in range(2):
                    for b in range(2):
                        e = e + 0.5 * g[a][b] * (Dr[a] * Dr[b] + Di[a] * Di[b])
            e = e - pot(u1, 0.0, u2 * math.cos(th), u2 * math.sin(th))
        return e * self.dA

    @staticmethod
    def _gamma(i):
        g12 = (-2.0 if i == 0 else 2.0) * SID["gamma12"]
        return [[2 * SID["gamma1"], g12], [g12, 2 * SID["gamma2"]]]

    @staticmethod
    def _cov(F, d, i):
        """Covariant derivatives of the two condensates along i: d p - i(-Q A) p as (real, imaginary) lists."""
        Q = SID["Q"]
        re = [d[2 + 2 * a][i] - Q * F[i] * F[3 + 2 * a] for a in range(2)]
        im = [d[3 + 2 * a][i] + Q * F[i] * F[2 + 2 * a] for a in range(2)]
        return re, im

    def gradient(self, F, raw=False):
        """dE/dphi per site; the flow's rows (projected, ring zeroed, the demag row scaled by -coup_mu) unless `raw`."""
        d = [self.jet(f) for f in F]
        g = torch.zeros_like(F)
        if self.t == "chiral":
            for a in range(3):
                g[a] = -(d[a][2] + d[a][3])
            g[0] += 2 * d[2][1] + d[3][0]
            g[1] += 2 * d[2][0] + d[3][1]
            g[2] -= 2 * d[0][1] + 2 * d[1][0] + self.ch + 2 * self.cK * F[2]
            g[3] = self.cmu * (d[0][0] + d[1][1]) - d[3][2] - d[3][3]
            if raw:
                g[3] /= -self.cmu
        elif self.t == "baby":
            dx, dy, xx, yy, xy = (torch.stack([v[k] for v in d]) for k in range(5))
            dot = lambda a, b: (a * b).sum(0)  # noqa: E731
            sA, sB = dot(xy, dy) - dot(yy, dx), dot(xy, dx) - dot(xx, dy)
            g = -(xx + yy) - self.kappa ** 2 * (xx * dot(dy, dy) + yy * dot(dx, dx) + dx * sA + dy * sB
                                                - 2 * xy * dot(dx, dy))
            g[2] -= 1.0
        elif self.t == "higgs":
            q = F[2] ** 2 + F[3] ** 2
            div, A2 = d[0][0] + d[1][1], F[0] ** 2 + F[1] ** 2
            g[0] = -d[0][3] + d[1][4] + F[2] * d[3][0] - F[3] * d[2][0] + F[0] * q
            g[1] = -d[1][2] + d[0][4] + F[2] * d[3][1] - F[3] * d[2][1] + F[1] * q
            g[2] = (-d[2][2] - d[2][3] + 2 * (F[0] * d[3][0] + F[1] * d[3][1]) + F[3] * div + A2 * F[2]
                    - 0.5 * (1 - q) * F[2])
            g[3] = (-d[3][2] - d[3][3] - 2 * (F[0] * d[2][0] + F[1] * d[2][1]) - F[2] * div + A2 * F[3]
                    - 0.5 * (1 - q) * F[3])
        else:
            self._sid_gradient(F, d, g)
        if raw:
            return g
        if self.t == "chiral":
            g *= self.mx * self.my
        if self.t in ("chiral", "baby"):
            g[:3] -= (g[:3] * F[:3]).sum(0, keepdim=True) * F[:3]
        return g

    def _sid_gradient(self, F, d, g):
        s, Q = SID, SID["Q"]
        pr, pi = (F[2], F[4]), (F[3], F[5])
        k2 = s["kappa"] ** 2
        g[0] = k2 * (d[1][4] - d[0][3])
        g[1] = k2 * (d[0][4] - d[1][2])
        for k in range(2):
            gm = self._gamma(k)
            for a in range(2):
                for b in range(2):
                    cur = pi[b] * d[2 + 2 * a][k] - pr[b] * d[3 + 2 * a][k]
                    g[k] -= Q * gm[a][b] * (cur - Q * F[k] * (pr[a] * pr[b] + pi[a] * pi[b]))
        # the condensate rows follow the flow's rows: the potential terms doubled, b4 terms as the flow has them
        n = [pr[a] ** 2 + pi[a] ** 2 for a in range(2)]
        al, be = (s["alpha1"], s["alpha2"]), (s["beta1"], s["beta2"])
        b3, b4 = s["beta3"], s["beta4"]
        for a in range(2):
            o = 1 - a
            w = pr[o] ** 2 - pi[o] ** 2
            g[2 + 2 * a] += 2 * pr[a] * (2 * al[a] + 4 * be[a] * n[a] + 2 * b3 * n[o])
            g[3 + 2 * a] += 2 * pi[a] * (2 * al[a] + 4 * be[a] * n[a] + 2 * b3 * n[o])
            g[2 + 2 * a] += 4 * b4 * (2 * pr[a] * w)
            g[3 + 2 * a] += 4 * b4 * (-2 * pi[a] * w)
        g[2] += 16 * b4 * F[3] * F[4] * F[5]
        g[3] += 16 * b4 * F[2] * F[4] * F[5]
        g[4] += 16 * b4 * F[2] * F[3] * F[5]
        g[5] += 16 * b4 * F[2] * F[3] * F[4]
        for i in range(2):
            gm = self._gamma(i)
            A, dA = F[i], d[i][i]
            for a in range(2):
                for b in range(2):
                    jr, ji = d[2 + 2 * b], d[3 + 2 * b]
                    g[2 + 2 * a] -= gm[a][b] * (jr[2 + i] - Q * Q * A * A * pr[b] - Q * (pi[b] * dA + 2 * A * ji[i]))
                    g[3 + 2 * a] -= gm[a][b] * (ji[2 + i] - Q * Q * A * A * pi[b] + Q * (pr[b] * dA + 2 * A * jr[i]))

    def flow(self, F, V, steps, E_prev):
        """`steps` arrested RK4 steps; returns (F, V, energies, errs)."""
        Es, errs, dt = [], [], self.dt
        for _ in range(steps):
            l1 = -dt * self.gradient(F)
            l2 = -dt * self.gradient(F + 0.5 * dt * V)
            l3 = -dt * self.gradient(F + 0.5 * dt * (V + 0.5 * l1))
            G = self.gradient(F + dt * (V + 0.5 * l2))
            l4 = -dt * G
            errs.append(float(G.max()))
            del G
            F = F + dt * V + dt / 6.0 * (l1 + l2 + l3)
            V = V + (l1 + 2 * l2 + 2 * l3 + l4) / 6.0
            del l1, l2, l3, l4
            if self.t in ("chiral", "baby"):
                F[:3] /= torch.sqrt((F[:3] ** 2).sum(0, keepdim=True))
                V[:3] -= (V[:3] * F[:3]).sum(0, keepdim=True) * F[:3]
            Es.append(float(self.energy_density(F).sum()))
            if Es[-1] > E_prev:
                V = torch.zeros_like(V)
            E_prev = Es[-1]
        return F, V, np.array(Es), np.array(errs)

    def skyrmion_density(self, F):
        d = [self.jet(F[a], False) for a in range(3)]
        c = torch.linalg.cross(torch.stack([v[0] for v in d]), torch.stack([v[1] for v in d]), dim=0)
        return (F[:3] * c).sum(0) * (self.dA / (4 * math.pi))


def exact(case, seed):
    theory, kind = case["theory"], case["kind"]
    dtype = _dtype(case["prec"])
    if kind == "sweep":
        fields, vels = [], []
        for i, n in enumerate(_sweep_sizes(case)):
            F = _field(theory, n, n, seed + 101 * i, dtype).double()
            F, V, _, _ = _Exact(theory, n, n, _sweep_kappa(i)).flow(F, torch.zeros_like(F), int(case["steps"]), math.nan)
            fields.append(F.reshape(-1))
            vels.append(V.reshape(-1))
        return fields + vels
    X, Y = case["X"], case["Y"]
    ex = _Exact(theory, X, Y)
    F = _field(theory, X, Y, seed, dtype).double()
    V = torch.zeros_like(F)
    if kind == "step":
        F, V, E, err = ex.flow(F, V, 1, 1e300)
        return dict(field=F.reshape(-1), velocity=V.reshape(-1), energy=float(E[0]), err=float(err[0]))
    if kind in ("relax", "advance", "frame"):
        F, V, E, err = ex.flow(F, V, int(case["steps"]), math.nan)
        out = dict(field=F.reshape(-1), velocity=V.reshape(-1))
        if kind == "relax":
            out.update(energy=E, err=err)
        if kind == "frame":
            out.update(density=ex.skyrmion_density(F).reshape(-1), jet=None, magnetization=None)
        return out
    if kind == "observe":
        dens = ex.energy_density(F)
        obs, cpl = dict(energy=float(dens.sum())), {}
        if theory in ("chiral", "baby"):
            obs["skyrmion_number"] = float(ex.skyrmion_density(F).sum())
        d = [ex.jet(f, False) for f in F]
        if theory == "chiral":
            obs["magnetic_charge"] = float(-(d[0][0] + d[1][1]).sum() * ex.dA)
            cpl["coup_K"] = float((1 - F[2] ** 2).sum() * ex.dA)
            cpl["coup_h"] = float((1 - F[2]).sum() * ex.dA)
            cpl["coup_mu"] = float((d[3][0] ** 2 + d[3][1] ** 2).sum() * ex.dA / (2 * ex.cmu ** 2))
            m = MAGNET
            cpl["B"] = cpl["coup_h"] * m["M"] * m["J"] / m["D"] ** 2
            cpl["K"] = cpl["coup_K"] * m["J"] / m["D"] ** 2
            cpl["D"] = -2.0 / m["D"] * (cpl["coup_K"] * ex.cK + cpl["coup_h"] * ex.ch + cpl["coup_mu"] * ex.cmu)
        elif theory == "baby":
            c = torch.linalg.cross(torch.stack([v[0] for v in d]), torch.stack([v[1] for v in d]), dim=0)
            cpl = dict(kappa=float((c * c).sum() * ex.dA), mpi=float(2 * (1 - F[2]).sum() * ex.dA))
        else:
            obs["vortex_number"] = float((d[1][0] - d[0][1]).sum() * ex.dA / (2 * math.pi))
            if theory == "higgs":
                cpl["Lambda"] = float(((1 - F[2] ** 2 - F[3] ** 2) ** 2).sum() / 8.0 * ex.dA)
        return dict(obs=obs, density=dens.reshape(-1), couplings=cpl)
    # grad
    return dict(energy=float(ex.energy_density(F).sum()), grad=(ex.gradient(F, raw=True) * ex.dA).reshape(-1))
