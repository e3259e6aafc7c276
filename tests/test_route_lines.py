"""Lattices at both sides of the node counts where lbm_step and lbm_adjoint pass
from the resident kernels to one launch per kernel (FP32 300,000 nodes; the
adjoint of a Bingham model 70,000 in FP64 and 90,000 in FP32, of a Newtonian one
160,000 in FP32): the results are those of one launch per kernel, which a
handle being profiled takes.  Steps to the bit in both precisions; gradients
within 2e-9 (FP64) and 2e-4 (FP32) of the entry and of the largest of its
kind, as in test_adjoint_levels."""

import numpy as np
import pytest

from test_adjoint_levels import run
from test_steps_resident import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("program", ["c3", "c6"])
@pytest.mark.parametrize("nx,ny", [(547, 546), (547, 547), (999, 299)])
def test_fp32_steps_at_the_line(pkg, cases, program, nx, ny):
    p, pin = build(cases, program, nx, ny, 2, 20.0, 1)
    p.series_every, p.series_capacity, p.series_particles = 2, 8, 2
    got = []
    for profiled in (False, True):
        s = pkg.Simulation(p)
        s.set_particles(pin)
        s.profile(profiled)
        s.step(12)
        s.step(3)
        assert s.kk == 15 and s.status() == 0
        f, om, ps = s.get_state()
        got.append({"f": f, "omega": om, "state": ps, "series": s.series()})
        s.close()
    for k, w in got[1].items():
        assert np.array_equal(got[0][k], w, equal_nan=True), k


@pytest.mark.parametrize("program,nx,ny,prec", [
    ("c6", 263, 263, 0), ("c6", 264, 264, 0), ("c6", 299, 299, 1), ("c6", 300, 299, 1),
    ("c1", 399, 399, 1), ("c1", 400, 399, 1)])
def test_gradients_at_the_line(pkg, cases, program, nx, ny, prec):
    p, pin = build(cases, program, nx, ny, 2 if program == "c6" else 1, 20.0, prec)
    p.contact_test = 0
    j, g, parts = run(pkg, p, pin, 8, 14, 4, False)
    jr, gr, partsr = run(pkg, p, pin, 8, 14, 4, True)
    assert j == jr and np.array_equal(parts, partsr)
    rtol = 2e-9 if prec == 0 else 2e-4
    for keys in (("tau_y",), ("nu",), ("rho_p",), ("x0", "y0")):
        scale = max(np.max(np.abs(np.atleast_1d(gr[k]))) for k in keys)
        for k in keys:
            a, b = np.atleast_1d(g[k]), np.atleast_1d(gr[k])
            assert np.all(np.isfinite(a)), k
            assert np.all(np.abs(a - b) <= rtol * (np.abs(b) + scale)), (k, a, b)


def test_gradient_that_fits_one_slot_set_only(pkg, cases):
    """Above the line a gradient keeps two sets of slots; a lattice that can
    step many steps per launch takes the one-set way where the second set does
    not fit in memory, and returns the same gradient (2e-9)."""
    torch = pytest.importorskip("torch")
    p, pin = build(cases, "c6", 280, 280, 2, 20.0, 0)
    p.contact_test, p.series_every = 0, 0
    every, n1 = 200, 404  # three segments; a slot is 10 planes of 281 rows
    want = run(pkg, p, pin, 400, n1, every, False)
    slot = 10 * 281 * 288 * 8
    sim = pkg.Simulation(p)
    sim.set_particles(pin)
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - int(1.5 * every * slot) - (64 << 20), dtype=torch.uint8,
                        device="cuda")
    try:
        j, g = sim.adjoint(400, n1, particle=1, checkpoint_every=every)
        parts = sim.particles()
    finally:
        del taken
        torch.cuda.empty_cache()
    assert sim.status() == 0
    sim.close()
    assert j == want[0] and np.array_equal(parts, want[2])
    for k, w in want[1].items():
        a, b = np.atleast_1d(g[k]), np.atleast_1d(w)
        scale = np.max(np.abs(b)) if k not in ("x0", "y0") else max(
            np.max(np.abs(want[1]["x0"])), np.max(np.abs(want[1]["y0"])))
        assert np.all(np.abs(a - b) <= 2e-9 * (np.abs(b) + scale)), k
