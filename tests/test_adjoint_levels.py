"""The adjoint of a small lattice (many reverse levels per launch, forward and
recompute by the resident multi-step kernel) against one launch per kernel: a
handle being profiled (lbm_profile) takes that path.

Both paths are within 1e-9 (FP64) and 1e-4 (FP32) of the exact derivative
(tests/test_adjoint.py), so they agree within twice that, of the entry and of
the largest entry of its kind (entries that vanish by symmetry, disks far from
the observed one).  The objective comes from the forward kernels, which share
their operations: bit for bit in FP64, 1e-5 in FP32."""

import numpy as np
import pytest

from test_steps_resident import build

pytestmark = pytest.mark.gpu

# (program, nx, ny, disks, diameter, n0, n1, checkpoint_every): no level, one,
# one per launch, launches of uneven lengths, all in one launch; one and two
# words of disks; a block of less than a warp's segments, several segments per
# warp; the largest lattice of the rule
CASES = [
    ("c1", 31, 40, 1, 6.0, 1, 1, 0),
    ("c1", 31, 40, 1, 6.0, 2, 2, 0),
    ("c6", 33, 64, 2, 6.0, 5, 12, 1),
    ("c6", 62, 95, 3, 8.0, 30, 41, 0),
    ("c3", 96, 131, 33, 8.0, 10, 23, 7),
    ("c3", 95, 130, 64, 8.0, 10, 21, 100),
    ("c1", 300, 400, 1, 20.0, 20, 30, 0),
    ("c6", 450, 880, 1, 24.0, 8, 16, 4),
]


def run(pkg, p, pin, n0, n1, every, profiled):
    sim = pkg.Simulation(p)
    sim.set_particles(pin)
    if profiled:
        sim.profile(True)
    j, g = sim.adjoint(n0, n1, particle=pin.shape[0] - 1, checkpoint_every=every)
    parts = sim.particles()
    sim.close()
    return j, g, parts


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("program,nx,ny,n,diam,n0,n1,every", CASES)
def test_levels_match_one_launch_per_kernel(pkg, cases, program, nx, ny, n, diam, n0, n1, every,
                                            prec):
    p, pin = build(cases, program, nx, ny, n, diam, prec)
    p.contact_test = 0
    j, g, parts = run(pkg, p, pin, n0, n1, every, False)
    jr, gr, partsr = run(pkg, p, pin, n0, n1, every, True)
    if prec == 0:
        assert j == jr
        assert np.array_equal(parts, partsr)
    else:
        assert abs(j - jr) <= 1e-5 * abs(jr)
    rtol = 2e-9 if prec == 0 else 2e-4
    for keys in (("tau_y",), ("nu",), ("rho_p",), ("x0", "y0")):
        scale = max(np.max(np.abs(np.atleast_1d(gr[k]))) for k in keys)
        for k in keys:
            a, b = np.atleast_1d(g[k]), np.atleast_1d(gr[k])
            assert np.all(np.isfinite(a)), k
            assert np.all(np.abs(a - b) <= rtol * (np.abs(b) + scale)), (k, a, b)
