"""Workloads of the library as its users run them, for timing and comparison.

A case is one chunk of a simulation program: some time steps through the
public API (``Simulation``, ``Batch``, ``Simulation.adjoint``) and the read of
what the program writes out after them.  ``listed()`` holds the shipped
programs and the configurations of the benchmark; ``draw()`` gives other
sizes, disk counts, rheologies and precisions of the same ranges; ``exact()``
is the same method in plain torch at 64 bits (autograd for the gradients).

Results of an FP32 run are kept in single precision (the populations carry no
more), results of an FP64 run in double.
"""

from __future__ import annotations

import importlib
import math

import numpy as np
import torch
import torch.utils.checkpoint

lbm = importlib.import_module("2d_nnf_lbm_b200")
programs = lbm.cases

F64, F32 = 0, 1  # lbm_params.precision


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # A patched Fortran program that keeps its own per-step output: one
        # library call per time step and the particle read after it, on the
        # smallest shipped lattice (the yield-stress program, 80 x 300).
        dict(name="yield_stepwise_f64", kind="run", program="c6", precision=F64, nx=80, ny=300,
             diam=20.0, disks=1, bn=0.5, steps=100, every=0, stepwise=True, stress=False,
             fields=""),
        # The plain method's configuration: the one-disk Newtonian program at
        # 200 x 600, in the chunks between two field outputs.
        dict(name="newton_plain_f64", kind="run", program="c1", precision=F64, nx=200, ny=600,
             diam=24.0, disks=1, bn=0.0, steps=1000, every=10, stepwise=False, stress=False,
             fields="ux uy rho"),
        # The multi-particle program at its shipped lattice, a record of every
        # disk at every step (what its driver writes).
        dict(name="sediment_512_f64", kind="run", program="c3", precision=F64, nx=512, ny=512,
             diam=16.0, disks=200, bn=0.0, steps=500, every=1, stepwise=False, stress=False,
             fields="ux uy"),
        # The oscillating-cylinder program at its shipped lattice (equilibrium
        # boundary, prescribed motion).
        dict(name="oscillate_f64", kind="run", program="c4", precision=F64, nx=1500, ny=1000,
             diam=50.0, disks=1, bn=0.0, steps=300, every=1, stepwise=False, stress=False,
             fields=""),
        # The headline configuration: 512 settling disks on 1024 x 2048, FP32
        # shifted populations, and the plain FP64 method on the same.
        dict(name="sediment_f32", kind="run", program="c3", precision=F32, nx=1024, ny=2048,
             diam=16.0, disks=512, bn=0.0, steps=1000, every=10, stepwise=False, stress=False,
             fields="ux"),
        dict(name="sediment_f64", kind="run", program="c3", precision=F64, nx=1024, ny=2048,
             diam=16.0, disks=512, bn=0.0, steps=500, every=1, stepwise=False, stress=False,
             fields="rho"),
        # The largest lattice the repository measures, with the most disks a
        # simulation may hold.
        dict(name="sediment_large_f32", kind="run", program="c3", precision=F32, nx=4096, ny=8192,
             diam=16.0, disks=4096, bn=0.0, steps=100, every=10, stepwise=False, stress=False,
             fields=""),
        # Viscoplastic settling at its configuration's size, the FP32 run and
        # the FP64 run it is compared with.
        dict(name="viscoplastic_f32", kind="run", program="c6", precision=F32, nx=800, ny=2400,
             diam=40.0, disks=1, bn=2.0, steps=1000, every=10, stepwise=False, stress=False,
             fields="rho"),
        dict(name="viscoplastic_f64", kind="run", program="c6", precision=F64, nx=800, ny=2400,
             diam=40.0, disks=1, bn=2.0, steps=250, every=10, stepwise=False, stress=False,
             fields="rho"),
        # The batched configuration: 256 Bingham runs of uneven widths.
        dict(name="batch_256_f32", kind="batch", precision=F32, sims=256, wmin=128, wmax=512,
             study=0, steps=64),
        # One gradient of a calibration loop on the adjoint configuration (a
        # shorter horizon), and a small Newtonian one in double precision.
        dict(name="adjoint_f32", kind="adjoint", program="c6", precision=F32, nx=400, ny=1200,
             diam=24.0, bn=5.0, n0=750, n1=1000),
        dict(name="adjoint_small_f64", kind="adjoint", program="c1", precision=F64, nx=100,
             ny=300, diam=16.0, bn=0.0, n0=300, n1=400),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["run", "batch", "adjoint"], [8, 1, 2])[0]
    precision = rng.choice([F64, F32])
    if kind == "batch":
        wmin = rng.randint(40, 160)
        return dict(kind="batch", precision=precision, sims=rng.randint(5, 96), wmin=wmin,
                    wmax=wmin + rng.randint(1, 200), study=rng.randint(1, 10 ** 6),
                    steps=rng.randint(16, 40))
    if kind == "adjoint":
        nodes = _log(rng, 2.0e4, 2.5e5)
        nx = int(math.sqrt(nodes / rng.uniform(2.0, 4.0)))
        n1 = rng.randint(100, 400)
        program = rng.choice(["c1", "c6"]) if precision == F32 else "c1"
        return dict(kind="adjoint", program=program, precision=precision, nx=nx,
                    ny=int(nodes / nx), diam=round(rng.uniform(8.0, nx / 5.0), 1),
                    bn=round(_log(rng, 0.1, 50.0), 3) if program == "c6" else 0.0,
                    n0=rng.randint(n1 // 2, n1), n1=n1)
    program = rng.choice(["c1", "c3", "c3", "c4", "c6", "c6"])
    nodes = _log(rng, 2.0e4, 6.0e6)
    aspect = {"c1": rng.uniform(2.0, 4.0), "c3": rng.uniform(0.8, 2.5),
              "c4": rng.uniform(0.5, 1.5), "c6": rng.uniform(2.5, 4.0)}[program]
    nx = int(math.sqrt(nodes / aspect))
    ny = int(nodes / nx)
    disks = 1
    diam = round(rng.uniform(nx / 12.0, nx / 5.0) if program != "c4" else nx / 25.0, 1)
    diam = min(max(diam, 8.0), 60.0)
    if program == "c3":
        diam = 16.0
        disks = min(4096, max(2, int(rng.uniform(0.02, 0.30) * 0.5 * nodes / 254.0)))
    steps = int(min(1500, max(60, rng.uniform(1.0e8, 3.0e8) / nodes)))
    stepwise = nodes < 2.0e5 and rng.random() < 0.3
    return dict(kind="run", program=program, precision=precision, nx=nx, ny=ny, diam=diam,
                disks=disks, bn=round(_log(rng, 0.1, 50.0), 3) if program == "c6" else 0.0,
                steps=min(steps, 200) if stepwise else steps,
                every=0 if stepwise else rng.choice([1, 1, 7, 10]), stepwise=stepwise,
                stress=program == "c6" and rng.random() < 0.3,
                fields="" if nodes > 3.0e5 else "ux uy" if program in ("c1", "c4") else "rho")


# ---- inputs -------------------------------------------------------------------
def _newton_input(case, rng):
    """The plain configuration (one disk, tau = 0.8, interface 2 lu) at the
    case's size, its gravity lowered for a larger disk so that the settling
    speed does not grow."""
    nx, ny, diam = case["nx"], case["ny"], case["diam"]
    p = programs.shipped_c1(nx, ny, diam)
    p.precision = case["precision"]
    p.nu = lbm.lbm2d.r4((0.8 - 0.5) / 3.0)
    p.zeta = 2.0
    p.gravity = programs.CFG1_GRAVITY * min(1.0, (24.0 / diam) ** 2)
    p.c_ij = lbm.lbm2d.glowinski_cij(1.5, 1.0, p.gravity, p.pi, diam)
    xy = [[nx * (0.5 + rng.choice([-1, 1]) * rng.uniform(0.05, 0.1)), 0.8 * ny + rng.uniform(-1, 1)]]
    return p, programs.pin_array(xy, diam, rng.uniform(1.3, 1.5))


def _run_input(case, seed):
    """Parameters and disks of a single run: the program's constants at the
    case's size, the disks' positions and densities from the seed."""
    rng = np.random.default_rng(seed)
    nx, ny, diam, prec = case["nx"], case["ny"], case["diam"], case["precision"]
    program = case["program"]
    if program == "c1":
        p, pin = _newton_input(case, rng)
    elif program == "c3":
        p, pin = programs.workload_cfg2(prec, nx, ny, case["disks"], seed)
    elif program == "c4":
        p, pin = programs.shipped_c4(nx, ny, diam, min(100.0, 0.05 * diam / 0.025))
        pin[:, 0:2] += rng.uniform(-2.0, 2.0, (1, 2))
    else:
        p, pin, _ = programs.workload_cfg3(prec, case["bn"], nx, ny, diam)
        p.tau_y *= rng.uniform(0.9, 1.1)
        pin[:, 0] += diam * rng.uniform(-0.4, 0.4)
        pin[:, 1] += rng.uniform(-1.0, 1.0)
    p.precision = prec
    p.series_every = case["every"]
    p.series_particles = case["disks"] if case["every"] else 0
    p.series_capacity = max(1, case["steps"])
    p.record_stress = 1 if case["stress"] else 0
    return p, pin


def _adjoint_input(case, seed):
    """Of a calibration loop: no history records beside the gradient."""
    rng = np.random.default_rng(seed)
    if case["program"] == "c1":
        p, pin = _newton_input(case, rng)
        p.series_every = 0
        return p, pin
    p, pin, _ = programs.workload_cfg5(case["precision"], case["bn"], case["nx"], case["ny"],
                                       case["diam"])
    p.tau_y *= rng.uniform(0.9, 1.1)
    p.series_every = 0
    pin[:, 0] += case["diam"] * rng.uniform(0.2, 0.5)
    pin[:, 1] += rng.uniform(-1.0, 1.0)
    return p, pin


def _batch_input(case, seed):
    """The batch study's generator over the case's widths; the seed varies the
    yield stresses and the disks' centres."""
    rng = np.random.default_rng(seed)
    runs = programs.workload_cfg4(case["precision"], case["sims"], case["study"])
    out = []
    for p, pin in runs:
        w = case["wmin"] + (p.nx - 128) * (case["wmax"] - case["wmin"]) // 384
        diam = max(8.0, w / 10.0)
        bn, rho_s = p.tau_y * pin[0, 6] / (p.nu * 0.78 * p.nu / pin[0, 6]), pin[0, 7]
        q, disk, _ = programs.workload_cfg5(case["precision"], bn, w, 3 * w, diam, rho_s)
        q.tau_y *= rng.uniform(0.9, 1.1)
        disk[:, 0] += diam * rng.uniform(-0.4, 0.4)
        q.series_every = 1
        q.series_particles = 1
        q.series_capacity = 2 * case["steps"]
        out.append((q, disk))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        p, pin = _adjoint_input(case, seed)
        return dict(case=case, params=p, pin=pin)
    if kind == "batch":
        runs = _batch_input(case, seed)
        b = lbm.Batch([p for p, _ in runs])
        for sim, (_, pin) in zip(b.sims, runs):
            sim.set_particles(pin)
        return dict(case=case, batch=b)
    p, pin = _run_input(case, seed)
    sim = lbm.Simulation(p)
    sim.set_particles(pin)
    return dict(case=case, sim=sim)


# ---- one pass -------------------------------------------------------------------
def _keep(case, a):
    return a.astype(np.float32) if case["precision"] == F32 else a


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        sim = lbm.Simulation(state["params"])
        sim.set_particles(state["pin"])
        value, grad = sim.adjoint(case["n0"], case["n1"])
        sim.close()
        out = {k: _keep(case, np.atleast_1d(np.asarray(v, dtype=np.float64)))
               for k, v in grad.items()}
        out["value"] = _keep(case, np.array([value]))
        return out
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        rec = np.stack([s.series() for s in b.sims])
        return dict(records=_keep(case, rec[:, :, 2:]), mean_density=_keep(case, rec[:, :, 1]),
                    particles=_keep(case, np.stack([s.particles() for s in b.sims])))
    sim = state["sim"]
    out = {}
    if case["stepwise"]:
        history = []
        for _ in range(case["steps"]):
            sim.step(1)
            history.append(sim.particles())
        out["history"] = _keep(case, np.stack(history))
    else:
        sim.step(case["steps"])
        rec = sim.series()
        out["records"] = _keep(case, rec[:, 2:].reshape(len(rec), -1, 12))
        out["mean_density"] = _keep(case, rec[:, 1])
        out["particles"] = _keep(case, sim.particles())
    for name in case["fields"].split():
        out[name] = _keep(case, sim.field(name))
    return out


# ---- the work of a pass -----------------------------------------------------------
def work(case):
    """Per node and step the nine populations (and a Bingham node's relaxation
    rate) are read once and written once; the gradient adds the recomputed
    forward step and the reverse step (state and adjoint fields read, adjoint
    fields written).  Operations: the moment transforms, the relaxation and
    the macroscopic variables (128 a node), 60 more with the viscosity."""
    size = 8 if case["precision"] == F64 else 4
    if case["kind"] == "batch":
        nodes = sum((p.nx + 1) * (p.ny + 1) for p, _ in _batch_input(case, 0))
        return dict(bytes=nodes * case["steps"] * 20 * size, flops=nodes * case["steps"] * 188)
    nodes = (case["nx"] + 1) * (case["ny"] + 1)
    if case["kind"] == "adjoint":
        return dict(bytes=nodes * case["n1"] * 70 * size, flops=nodes * case["n1"] * 800)
    bingham = case["program"] == "c6"
    per = (20 if bingham else 18) * size
    return dict(bytes=nodes * case["steps"] * per,
                flops=nodes * case["steps"] * (188 if bingham else 128))


# ---- the method in plain torch at 64 bits -------------------------------------------
CX = [0, 1, 0, -1, 0, 1, -1, -1, 1]
CY = [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP = [0, 3, 4, 1, 2, 7, 8, 5, 6]
MOMENTS = [[1, 1, 1, 1, 1, 1, 1, 1, 1], [-4, -1, -1, -1, -1, 2, 2, 2, 2],
           [4, -2, -2, -2, -2, 1, 1, 1, 1], [0, 1, 0, -1, 0, 1, -1, -1, 1],
           [0, -2, 0, 2, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1],
           [0, 0, -2, 0, 2, 1, 1, -1, -1], [0, 1, -1, 1, -1, 0, 0, 0, 0],
           [0, 0, 0, 0, 0, 1, -1, 1, -1]]


class Method:
    """The time step of one simulation: populations f[9, NY+1, NX+1] after
    collision, a node relaxation rate and the disks' state."""

    def __init__(self, p, pin, nu=None, tau_y=None):
        self.p = p
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.M = t(MOMENTS)
        self.Minv = torch.linalg.inv(self.M) * (36.0 * p.d_mrt)
        self.nu = t(p.nu) if nu is None else nu
        self.tau_y = t(p.tau_y) if tau_y is None else tau_y
        self.bingham = p.rheology == lbm.lbm2d.LBM_BINGHAM
        self.diam = t(pin[:, 6])
        self.cx, self.cy = t(CX).view(9, 1, 1), t(CY).view(9, 1, 1)
        reach = int(math.ceil(0.5 * float(pin[:, 6].max()) + 0.5 * p.zeta)) + 1
        r = torch.arange(-reach, reach + 1, device=self.dev)
        self.wj, self.wi = (w.reshape(-1) for w in torch.meshgrid(r, r, indexing="ij"))

    def start(self, pin):
        """INITIALIZE: fluid at rest, and the collision of step 1."""
        p = self.p
        t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        zero = torch.zeros(p.ny + 1, p.nx + 1, dtype=torch.float64, device=self.dev)
        f = self.equilibrium(zero + p.rho0, zero, zero)
        omega = zero + 1.0 / (3.0 * self.nu + 0.5)
        disk = {"x": t(pin[:, 0:2]), "v": t(pin[:, 3:6]), "angle": t(pin[:, 2])}
        disk["old"] = torch.zeros_like(disk["v"])
        disk["force"] = torch.zeros_like(disk["v"])
        self.rho, self.ux, self.uy = zero + p.rho0, zero, zero
        f, omega = self.collide(f, zero + p.rho0, zero, zero, zero, zero, omega)
        return f, omega, disk

    def equilibrium(self, rho, ux, uy):
        w = [self.p.w_init[0 if k == 0 else (1 if k < 5 else 2)] for k in range(9)]
        uu = ux * ux + uy * uy
        out = []
        for k in range(9):
            c = CX[k] * ux + CY[k] * uy
            b = 2.0 + 6.0 * c + 9.0 * c * c - 3.0 * uu
            out.append(w[k] * rho * (b if k < 5 else 0.5 * b))
        return torch.stack(out)

    def collide(self, f, rho, ux, uy, gx, gy, omega):
        p = self.p
        m = torch.tensordot(self.M, f, dims=1)
        uu = ux * ux + uy * uy
        eq = [rho, rho * (3 * uu - 2), rho * (1 - 3 * uu), rho * ux, -rho * ux, rho * uy,
              -rho * uy, rho * (ux * ux - uy * uy), rho * ux * uy]
        fx, fy = rho * gx, rho * gy
        fu = fx * ux + fy * uy
        mf = [None, 6 * fu, -6 * fu, fx, -fx, fy, -fy, 2 * (fx * ux - fy * uy), fy * ux + fx * uy]
        sq = 8 * (2 - omega) / (8 - omega) if p.rate_set == lbm.lbm2d.LBM_RATES_Q_OF_OMEGA else p.s_q
        s = [0.0, p.s_e, p.s_eps, 0.0, sq, 0.0, sq, omega, omega]
        new = []
        for k in range(9):
            v = m[k]
            if k in (3, 5):
                v = v + mf[k]
            elif k:
                v = v - s[k] * (m[k] - eq[k]) + (1 - 0.5 * s[k]) * mf[k]
            new.append(v)
        out = torch.tensordot(self.Minv, torch.stack(new), dims=1)
        if not self.bingham:
            return out, omega
        y1, y7, y8 = p.s_e * (m[1] - eq[1]), omega * (m[7] - eq[7]), omega * (m[8] - eq[8])
        kap, gu = 36.0 * p.d_mrt, gx * ux + gy * uy
        d11 = -kap * (0.25 * y1 + 0.75 * y7) + 0.75 * ((omega - p.s_e) * gu - 2 * omega * gx * ux)
        d22 = -kap * (0.25 * y1 - 0.75 * y7) + 0.75 * ((omega - p.s_e) * gu - 2 * omega * gy * uy)
        d12 = -1.5 * kap * y8 - 0.75 * omega * (gx * uy + gy * ux)
        d11, d22, d12 = d11 / rho, d22 / rho, d12 / rho
        g2 = 2 * (d11 * d11 + d22 * d22 + 2 * d12 * d12)
        some = g2 > 0
        x = p.m_pap * torch.where(some, torch.sqrt(torch.where(some, g2, torch.ones_like(g2))),
                                  torch.zeros_like(g2))
        small = x < 1e-5
        xs = torch.where(small, torch.ones_like(x), x)
        ratio = torch.where(small, 1 - 0.5 * x + x * x / 6, -torch.expm1(-xs) / xs)
        nua = self.nu + self.tau_y * p.m_pap * ratio
        return out, 1.0 / (3.0 * nua / rho + 0.5)

    def stream(self, f):
        """Pull streaming and the boundary conditions of the populations f."""
        p, out = self.p, []
        for k in range(9):
            t = torch.roll(f[k], (CY[k], CX[k]), (0, 1)) if k else f[k].clone()
            if CY[k]:
                t[0 if CY[k] > 0 else -1, :] = f[k][0 if CY[k] > 0 else -1, :]
            if CX[k]:
                t[:, 0 if CX[k] > 0 else -1] = f[k][:, 0 if CX[k] > 0 else -1]
            out.append(t)
        if p.bc == lbm.lbm2d.LBM_BC_EQUILIBRIUM:
            r, x, y = self.rho, self.ux, self.uy
            put = lambda g, at, frm: [t.__setitem__(at, v) for t, v in  # noqa: E731
                                      zip(g, self.equilibrium(r[frm], x[frm], y[frm]))]
            inner = slice(1, -1)
            for at, frm in (((0, inner), (1, inner)), ((-1, inner), (-2, inner)),
                            ((inner, 0), (inner, 1)), ((inner, -1), (inner, -2)),
                            ((0, 0), (1, 1)), ((0, -1), (1, -2)), ((-1, 0), (-2, 1)),
                            ((-1, -1), (-2, -2))):
                put(out, at, frm)
            return torch.stack(out)
        inner = slice(1, -1)
        sides = [((-1, inner), 4, 8, 7, 6, 5, 1, 3), ((0, inner), 2, 5, 6, 7, 8, 1, 3),
                 ((inner, 0), 1, 5, 8, 7, 6, 2, 4), ((inner, -1), 3, 6, 7, 8, 5, 2, 4)]
        for at, n, a, b, oa, ob, t0, t1 in sides:
            if p.bc == lbm.lbm2d.LBM_BC_HALFWAY_BB:
                for k in (n, a, b):
                    out[k][at] = f[OPP[k]][at]
            else:  # Zou-He with resting walls
                d = 0.5 * (out[t0][at] - out[t1][at])
                out[n][at] = out[OPP[n]][at].clone()
                out[a][at] = out[oa][at] - d
                out[b][at] = out[ob][at] + d
        for at, ks in (((0, 0), (1, 5, 2)), ((-1, 0), (1, 8, 4)), ((-1, -1), (3, 7, 4)),
                       ((0, -1), (2, 6, 3))):
            for k in ks:
                out[k][at] = f[OPP[k]][at]
        return torch.stack(out)

    def repulsion(self, x):
        p = self.p
        force = torch.zeros_like(x)
        if p.wall_model != lbm.lbm2d.LBM_WALL_NONE:
            d, z = self.diam, p.rep_zeta
            if p.wall_model == lbm.lbm2d.LBM_WALL_MIRROR:
                es = [(1, 2 * x[:, 1]), (0, 2 * x[:, 0] - 2 * p.nx),
                      (1, 2 * x[:, 1] - p.wall_mirror_top), (0, 2 * x[:, 0] - p.wall_mirror_left)]
            else:
                es = [(1, x[:, 1] + 0.5 * d), (0, x[:, 0] - p.nx - 0.5 * d),
                      (1, x[:, 1] - p.ny - 0.5 * d), (0, x[:, 0] + 0.5 * d)]
            cols = [0.0, 0.0]
            for axis, e in es:
                r = e.abs()
                q = (r - d - z) / z
                g = p.eps_w * p.c_ij * q * q
                g = g + torch.where(r <= d, p.e_w * p.c_ij * (d - r) / z, torch.zeros_like(r))
                cols[axis] = cols[axis] + torch.where(r > d + z, torch.zeros_like(r), g * torch.sign(e))
            force = torch.stack(cols, 1)
        if len(x) > 1:
            e = x[:, None, :] - x[None, :, :]
            r = torch.sqrt((e * e).sum(-1) + torch.eye(len(x), dtype=x.dtype, device=x.device))
            c = 0.5 * (self.diam[:, None] + self.diam[None, :])
            z = p.rep_zeta
            q = (r - c - z) / z
            g = p.eps_p * p.c_ij * q * q
            g = g + torch.where(r <= c, p.e_p * p.c_ij * (c - r) / z, torch.zeros_like(r))
            g = torch.where(r > c + z, torch.zeros_like(r), g)
            g = g * (1 - torch.eye(len(x), dtype=x.dtype, device=x.device))
            force = force + (g / r).unsqueeze(-1).mul(e).sum(1)
        return force

    def move(self, disk, rho_p, step):
        """Newton-Euler with the internal-mass term, or the prescribed motion."""
        p = self.p
        mass = rho_p * p.pi * (0.5 * self.diam) ** 2
        inert = 0.5 * mass * (0.5 * self.diam) ** 2
        mi = torch.stack([mass, mass, inert], 1)
        rr = (p.rho0 / rho_p).unsqueeze(1)
        col = self.repulsion(disk["x"])
        v, old = disk["v"], disk["old"]
        if p.motion == lbm.lbm2d.LBM_MOTION_OSCILLATE:
            new = torch.zeros_like(v)
            new[:, 0] = -p.osc_u * math.cos(2.0 * p.pi * step / p.osc_period)
            fin = rr * mi * (new - v)
        else:
            fin = rr * mi * (v - old)
            acc = torch.zeros_like(v)
            acc = torch.cat([acc[:, :1], ((1.0 - p.rho0 / rho_p) * p.gravity).unsqueeze(1),
                             acc[:, 2:]], 1)
            new = v + (disk["force"] + fin + torch.cat([col, acc[:, 2:]], 1)) / mi + acc
        x = disk["x"] + 0.5 * (new[:, 0:2] + v[:, 0:2])
        angle = disk["angle"] + 0.5 * (new[:, 2] + v[:, 2]) if p.integrate_angle else disk["angle"]
        return dict(x=x, v=new, old=v, angle=angle, force=disk["force"], fin=fin, col=col,
                    mass=mass, inert=inert)

    def step(self, f, omega, disk, rho_p, step):
        p = self.p
        disk = self.move(disk, rho_p, step)
        F = self.stream(f)
        rho = F.sum(0)
        ux, uy = (self.cx * F).sum(0) / rho, (self.cy * F).sum(0) / rho
        x, v = disk["x"], disk["v"]
        c = torch.floor(x.detach()).long()
        i, j = c[:, 0:1] + self.wi, c[:, 1:2] + self.wj
        inside = (i >= 0) & (i <= p.nx) & (j >= 0) & (j <= p.ny)
        n = (j * (p.nx + 1) + i).clamp(0, rho.numel() - 1)
        di, dj = i - x[:, 0:1], j - x[:, 1:2]
        d = 0.5 * self.diam[:, None] - torch.sqrt(di * di + dj * dj)
        phi = 0.5 * (torch.sin(p.pi * d.clamp(-0.5 * p.zeta, 0.5 * p.zeta) / p.zeta) + 1.0)
        phi = torch.where(d >= 0.5 * p.zeta, torch.ones_like(d), phi)
        phi = torch.where((d > -0.5 * p.zeta) & inside, phi, torch.zeros_like(d))
        ur, uxn, uyn = rho.reshape(-1)[n], ux.reshape(-1)[n], uy.reshape(-1)[n]
        upx, upy = v[:, 0:1] - v[:, 2:3] * dj, v[:, 1:2] + v[:, 2:3] * di
        ex, ey, w = uxn - upx, uyn - upy, ur * phi
        disk["force"] = torch.stack([(w * ex).sum(1), (w * ey).sum(1),
                                     (w * (di * ey - dj * ex)).sum(1)], 1)
        # the highest-index disk with phi > 0 sets the body force of a node
        which = torch.arange(len(x), device=self.dev)[:, None].expand_as(n)
        hit = phi > 0
        last = torch.full((rho.numel(),), -1, dtype=torch.long, device=self.dev)
        last.scatter_reduce_(0, n[hit], which[hit], "amax")
        wins = hit & (last[n] == which)
        flat = torch.zeros(2, rho.numel(), dtype=torch.float64, device=self.dev)
        g = flat.index_put((torch.zeros_like(n[wins]), n[wins]), -(phi * ex)[wins])
        g = g.index_put((torch.ones_like(n[wins]), n[wins]), -(phi * ey)[wins])
        gx, gy = g[0].view_as(rho), g[1].view_as(rho)
        ux, uy = ux + 0.5 * gx, uy + 0.5 * gy
        self.rho, self.ux, self.uy = rho, ux, uy
        f, omega = self.collide(F, rho, ux, uy, gx, gy, omega)
        return f, omega, disk


def _columns(disk):
    z = torch.stack([disk["x"][:, 0], disk["x"][:, 1], disk["angle"]], 1)
    return torch.cat([z, disk["v"]], 1)


def _particles(disk):
    return torch.cat([_columns(disk), disk["force"], disk["col"], disk["fin"],
                      disk["mass"][:, None], disk["inert"][:, None]], 1)


@torch.no_grad()
def _exact_run(p, pin, case):
    m = Method(p, pin)
    rho_p = torch.as_tensor(pin[:, 7], dtype=torch.float64, device=m.dev)
    f, omega, disk = m.start(pin)
    records, density, history = [], [], []
    for k in range(1, case["steps"] + 1):
        before = disk["force"]
        f, omega, disk = m.step(f, omega, disk, rho_p, k)
        if case.get("stepwise"):
            history.append(_particles(disk))
        elif k % p.series_every == 0:
            records.append(torch.cat([_columns(disk), before, disk["fin"]], 1))
            density.append(m.rho.mean())
    if case.get("stepwise"):
        out = dict(history=torch.stack(history))
    else:
        out = dict(records=torch.stack(records), mean_density=torch.stack(density),
                   particles=_particles(disk))
    for name in case.get("fields", "").split():
        out[name] = getattr(m, name)
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_adjoint(p, pin, case):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    leaf = lambda v: torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)  # noqa: E731
    nu, tau_y, rho_p = leaf(p.nu), leaf(p.tau_y), leaf(pin[:, 7])
    x = leaf(pin[:, 0:2])
    m = Method(p, pin, nu, tau_y)
    f, omega, disk = m.start(pin)
    disk["x"] = x + 0.0
    state = (f, omega, disk["x"], disk["v"], disk["old"], disk["angle"], disk["force"])
    n0, n1 = case["n0"], case["n1"]

    def segment(lo, hi, f, omega, x, v, old, angle, force):
        d, total = dict(x=x, v=v, old=old, angle=angle, force=force), 0.0 * x[0, 0]
        for k in range(lo, hi):
            f, omega, d = m.step(f, omega, d, rho_p, k)
            if k >= n0:
                total = total + d["v"][0, 1]
        return (f, omega, d["x"], d["v"], d["old"], d["angle"], d["force"], total)

    size = max(4, min(40, int(2.0e10 / (1600.0 * f.numel() / 9))))
    value = torch.zeros((), dtype=torch.float64, device=dev)
    for lo in range(1, n1 + 1, size):
        *state, part = torch.utils.checkpoint.checkpoint(
            segment, lo, min(lo + size, n1 + 1), *state, use_reentrant=False)
        value = value + part
    value = value / (n1 - n0 + 1)
    grad = torch.autograd.grad(value, [tau_y, nu, rho_p, x], allow_unused=True)
    grad = [torch.zeros_like(tau_y) if g is None else g for g in grad]  # Newtonian: no tau_y
    a = lambda t: np.atleast_1d(t.detach().cpu().numpy())  # noqa: E731
    return dict(value=a(value), tau_y=a(grad[0]), nu=a(grad[1]), rho_p=a(grad[2]),
                x0=a(grad[3][:, 0]), y0=a(grad[3][:, 1]))


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(*_adjoint_input(case, seed), case)
    if case["kind"] == "batch":
        if case["sims"] * case["steps"] > 4096:
            return None
        got = [_exact_run(p, pin, dict(steps=case["steps"])) for p, pin in _batch_input(case, seed)]
        out = {k: np.stack([g[k] for g in got]) for k in ("records", "mean_density", "particles")}
        out["records"] = out["records"].reshape(len(got), case["steps"], -1)
        return out
    return _exact_run(*_run_input(case, seed), case)
