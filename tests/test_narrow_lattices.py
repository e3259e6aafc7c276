"""Narrow, tall lattices below the resident kernel's node limit: a row takes a
32-node segment however narrow it is, so above a number of rows the blocks'
segment queues (STEPS_MAX_SEGS a block) cannot hold them and the particle and
step kernels take the steps, as a handle being profiled does anyway.  FP64
results are those of that path bit for bit on both sides of the line, which
lies at 75,776 rows on 148 SMs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(pkg, p, pin, profiled):
    s = pkg.Simulation(p)
    try:
        s.set_particles(pin)
        s.profile(profiled)
        s.step(5)
        s.step(2)
        assert s.kk == 7 and s.status() == 0
        return {"particles": s.particles(), "uy": s.field("uy"), "rho": s.field("rho"),
                "series": s.series()}
    finally:
        s.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny", [(2, 75774), (2, 75776), (2, 100000), (4, 79990), (31, 12400)])
def test_narrow_lattice_steps(pkg, cases, nx, ny, precision):
    p = cases.shipped_c1(nx, ny, 2.0)
    p.precision = precision
    p.gravity = -1e-5
    p.wall_model = 2  # the walls are within the disk's repulsion range
    p.series_every = 1
    pin = cases.pin_array([[1.0, ny - 8.3]], 1.0, 1.25, uvw=[[0.0, -1e-3, 1e-3]])
    got, want = run(pkg, p, pin, False), run(pkg, p, pin, True)
    for k, w in want.items():
        if precision == 0:
            assert np.array_equal(got[k], w, equal_nan=True), k
        else:  # forces and fields relative to their scale, as in test_steps_resident
            a, b = np.nan_to_num(got[k]), np.nan_to_num(w)
            assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b)), k


def test_narrow_lattice_adjoint(pkg, cases):
    """lbm_adjoint above the line: the gradient of the one-launch-per-kernel
    path (the same kernels; its sums are atomics, 1e-9 as in test_adjoint)."""
    p = cases.shipped_c1(3, 80000, 2.0)
    p.gravity = -1e-5
    p.wall_model = 2
    p.series_every = 0
    pin = cases.pin_array([[1.6, 40000.2]], 1.0, 1.25)
    out = []
    for profiled in (False, True):
        s = pkg.Simulation(p)
        s.set_particles(pin)
        s.profile(profiled)
        out.append(s.adjoint(2, 4))
        assert s.status() == 0
        s.close()
    (j, g), (jr, gr) = out
    assert j == jr
    for k in gr:
        a, b = np.atleast_1d(g[k]), np.atleast_1d(gr[k])
        assert np.all(np.isfinite(a))
        assert np.all(np.abs(a - b) <= 1e-9 * np.maximum(np.abs(b), np.max(np.abs(b)))), k
