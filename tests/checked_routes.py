"""Small runs through each route of a time step and of the adjoint, shared by
tests/test_checked_routes.py (ordinary library, in process) and by a child
process that loads the checked library (LBM2D_LIBRARY):

    python tests/checked_routes.py OUT.npz

The cases of tests/checked_cases.py are all small enough for the resident
kernels; here they run with one launch per kernel too (a handle being
profiled): the step kernel's listed tiles and staged omega, the particle
kernel's pair and tile lists and history records, the adjoint's lattice and
particle kernels.  The resident kernels run with one and several warps of
disks, the equilibrium boundary's ring, a history ring that wraps, more steps
than one launch takes, and 64 disks in the adjoint.
"""

from __future__ import annotations

import importlib
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, ROOT)
sys.path.insert(0, HERE)
sys.path.insert(0, os.path.join(HERE, "golden"))

GRADS = ("tau_y", "nu", "rho_p", "x0", "y0")


def run_cases(pkg) -> dict:
    import adjoint_cases as ac
    from test_steps_resident import build

    cases = pkg.cases
    res = {}

    def steps(name, p, pin, n, profiled):
        sim = pkg.Simulation(p)
        sim.set_particles(pin)
        sim.profile(profiled)
        sim.step(n)
        sim.step(3)
        res.update({f"{name}_particles": sim.particles(), f"{name}_ux": sim.field("ux"),
                    f"{name}_series": sim.series(), f"{name}_status": np.array(sim.status())})
        sim.close()

    def gradient(name, p, pin, n0, n1, every, profiled):
        sim = pkg.Simulation(p)
        sim.set_particles(pin)
        sim.profile(profiled)
        j, g = sim.adjoint(n0, n1, checkpoint_every=every)
        res[f"{name}_j"] = np.array(j)
        res[f"{name}_grad"] = np.concatenate([np.atleast_1d(np.asarray(g[k])) for k in GRADS])
        res[f"{name}_status"] = np.array(sim.status())
        sim.close()

    for prec in (0, 1):
        # as tests/checked_cases.py, with one launch per kernel
        p, pin = cases.workload_cfg2(prec, 256, 512, 100)
        steps(f"two_sed{prec}", p, pin, 150, True)
        p, disk = cases.shipped_c6(80, 240)
        p.precision, p.record_stress, p.series_every, p.series_particles = prec, 1, 5, 1
        steps(f"two_c6{prec}", p, disk, 150, True)
        # the resident kernel
        for program, nx, ny, n, diam, every, cap, stress in (
                ("c6", 32, 65, 1, 8.0, 3, 5, 1), ("c4", 63, 47, 1, 9.0, 2, 6, 0),
                ("c3", 96, 131, 33, 8.0, 7, 3, 1), ("c3", 300, 301, 256, 12.0, 1, 40, 0)):
            p, pin = build(cases, program, nx, ny, n, diam, prec)
            p.record_stress, p.series_every, p.series_capacity = stress, every, cap
            p.series_particles = n
            steps(f"res{prec}_{program}_{n}", p, pin, 60, False)
        p, pin = build(cases, "c1", 31, 40, 1, 6.0, prec)
        p.series_every = 0
        steps(f"res{prec}_long", p, pin, 1100, False)
        p, pin, n0, n1 = ac.build(cases, "c3_pair")
        gradient(f"two_adj{prec}", p.copy(precision=prec), pin, n0, n1, 0, True)
        p, pin = build(cases, "c3", 95, 130, 64, 8.0, prec)
        p.contact_test = 0
        gradient(f"res{prec}_adj64", p, pin, 10, 21, 7, False)
    res["checked_build"] = np.array(int(pkg.load_library().lbm_checked_build()))
    return res


if __name__ == "__main__":
    pkg = importlib.import_module("2d_nnf_lbm_b200")
    np.savez(sys.argv[1], **run_cases(pkg))
