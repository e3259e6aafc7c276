"""The resident multi-step kernel (small lattices, lbm_step) against the
particle and step kernels on the same runs: a handle being profiled
(lbm_profile) steps with those two kernels, one step per launch.

FP64 runs agree bit for bit (the same operations in the same order, force and
mass sums exact); FP32 runs within 1e-6 of each quantity's scale, forces
within 1e-5 (the two kernels may contract products differently, a few 2^-24
per step of populations whose sums the forces are)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid_disks(cases, n, diam, nx, ny, gap=1.0):
    """n disks of one size in rows from the top left corner, each turning."""
    per = max(1, int((nx - gap) // (diam + gap)))
    k = np.arange(n)
    xy = np.stack([0.5 * diam + gap + (diam + gap) * (k % per),
                   ny - 0.5 * diam - gap - (diam + gap) * (k // per)], axis=1)
    uvw = np.zeros((n, 3))
    uvw[:, 0] = 1e-3 * ((k % 3) - 1)
    uvw[:, 2] = 1e-4 * ((k % 5) - 2)
    return cases.pin_array(xy, diam, 1.2 + 0.01 * (k % 7), uvw=uvw)


def build(cases, program, nx, ny, n, diam, prec):
    if program == "c1":
        p = cases.shipped_c1(nx, ny, max(diam, 1.0))
        p.gravity = -1e-5
        p.contact_test = 0
    elif program == "c3":
        p = cases.shipped_c3(nx, ny)
        p.gravity = -5e-5
        p.rep_zeta = 2.0
    elif program == "c4":
        p, _ = cases.shipped_c4(nx, ny, max(diam, 4.0), 2.0, 500.0)
    else:
        p, _ = cases.shipped_c6(nx, ny)
    p.precision = prec
    return p, grid_disks(cases, n, diam, nx, ny) if n else None


# lattice sizes at the edges of a 32-node segment and of a block's share, one
# disk warp / several (1, 32, 33, 256 disks), none, every boundary kind, the
# stress record, a history ring that wraps, and the largest lattice of the rule
CASES = [
    ("c1", 2, 2, 0, 0.0, 1, 4, 0),
    ("c1", 31, 40, 1, 6.0, 1, 7, 0),
    ("c6", 32, 65, 1, 8.0, 3, 5, 1),
    ("c6", 33, 64, 2, 6.0, 1, 64, 0),
    ("c4", 63, 47, 1, 9.0, 2, 6, 0),
    ("c3", 95, 130, 32, 8.0, 1, 11, 0),
    ("c3", 96, 131, 33, 8.0, 7, 3, 1),
    ("c3", 300, 301, 256, 12.0, 1, 40, 0),
    ("c1", 631, 631, 0, 0.0, 10, 8, 0),
]


def read_all(s):
    f, om, ps = s.get_state()
    out = {"f": f, "omega": om, "state": ps, "particles": s.particles(),
           "ux": s.field("ux"), "uy": s.field("uy"), "phi": s.field("phi")}
    if s.params.record_stress:
        out["tau12"] = s.field("tau12")
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("program,nx,ny,n,diam,every,cap,stress", CASES)
def test_resident_steps_match_one_step_per_launch(pkg, cases, program, nx, ny, n, diam, every,
                                                  cap, stress, precision):
    p, pin = build(cases, program, nx, ny, n, diam, precision)
    p.series_every, p.series_capacity, p.series_particles = every, cap, n
    p.record_stress = stress
    runs = []
    for mode in ("resident", "profiled", "mixed"):
        s = pkg.Simulation(p)
        try:
            if pin is not None:
                s.set_particles(pin)
            rec = []
            for k, steps in enumerate((1, 2, 25, 30)):
                s.profile(mode == "profiled" or (mode == "mixed" and k % 2 == 1))
                s.step(steps)
                if k != 1:
                    rec.append(s.series())
            assert s.kk == 58 and s.status() == 0
            got = read_all(s)
            got["series"] = np.concatenate(rec)
            runs.append(got)
        finally:
            s.close()
    want = runs[1]
    assert want["series"].shape[0] == 58 // every
    for got in (runs[0], runs[2]):
        for k, w in want.items():
            g = got[k]
            assert g.shape == w.shape, k
            if precision == 0:
                assert np.array_equal(g, w, equal_nan=True), k
            elif w.size and k not in ("state", "particles", "series"):
                assert np.max(np.abs(g - w)) <= 1e-6 * max(np.max(np.abs(w)), 1e-300), k
            elif w.size:
                # columns: positions, velocities, forces ... each by its scale
                g2, w2 = g.reshape(g.shape[0], -1), w.reshape(w.shape[0], -1)
                ok = np.isfinite(w2)
                scale = np.max(np.abs(np.where(ok, w2, 0.0)), axis=0)
                rel = 1e-5 * np.maximum(scale, 1e-9)
                assert np.all(np.abs(np.where(ok, g2 - w2, 0.0)) <= rel), k


def test_resident_handles_interleave(pkg, cases):
    """Two handles whose resident launches overlap in time on their own
    streams give the runs they give alone."""
    p, pin = build(cases, "c3", 120, 140, 20, 8.0, 0)
    p.series_every = 0
    alone = []
    for _ in range(2):
        s = pkg.Simulation(p)
        s.set_particles(pin)
        s.step(200)
        alone.append(s.particles())
        s.close()
    a, b = pkg.Simulation(p), pkg.Simulation(p)
    a.set_particles(pin)
    b.set_particles(pin)
    for _ in range(20):
        a.step(10)
        b.step(10)
    assert np.array_equal(a.particles(), alone[0])
    assert np.array_equal(b.particles(), alone[1])
    a.close()
    b.close()


@pytest.mark.parametrize("program,nx,ny,n,diam", [("c6", 32, 65, 1, 8.0), ("c3", 96, 131, 33, 8.0)])
def test_calls_of_one_step_mix_with_longer_ones(pkg, cases, program, nx, ny, n, diam):
    """A call of one step takes the two kernels while the tile lists are up to
    date, the resident kernel after a longer call: FP64 bit for bit the same
    as one call."""
    p, pin = build(cases, program, nx, ny, n, diam, 0)
    p.series_every = 0
    got = []
    for calls in ((40,), (1, 1, 1, 12, 1, 1, 2, 20, 1), (1,) * 40):
        s = pkg.Simulation(p)
        s.set_particles(pin)
        for k in calls:
            s.step(k)
        assert s.kk == 40 and s.status() == 0
        got.append(read_all(s))
        s.close()
    for g in got[1:]:
        for k, w in got[0].items():
            assert np.array_equal(g[k], w, equal_nan=True), k
