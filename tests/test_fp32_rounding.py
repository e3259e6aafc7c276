"""FP32 runs round alike in every kernel: the FP32 translation unit is built
with --fmad=false and writes out what is fused, so the kernels that share an
operation give the same bits -- the step kernel, the resident multi-step kernel
and both batch kernels (the autotuner chooses between those by time, so a
batch's results may not depend on the choice)."""

import numpy as np
import pytest

from test_steps_resident import CASES, build, read_all

pytestmark = pytest.mark.gpu


def turning(pin):
    """The same disks, turning fast enough for the rigid velocity's rounding
    to reach the force sums."""
    if pin is not None:
        pin = pin.copy()
        pin[:, 5] = 3e-3 * (1.0 + 0.1 * (np.arange(len(pin)) % 5))
    return pin


def assert_same(got, want, what):
    for k, w in want.items():
        assert np.array_equal(got[k], w, equal_nan=True), (what, k)


@pytest.mark.parametrize("program,nx,ny,n,diam,every,cap,stress", CASES)
def test_resident_steps_give_the_step_kernels_bits(pkg, cases, program, nx, ny, n, diam, every,
                                                   cap, stress):
    p, pin = build(cases, program, nx, ny, n, diam, 1)
    pin = turning(pin)
    p.series_every, p.series_capacity, p.series_particles = every, cap, n
    p.record_stress = stress
    runs = []
    for profiled in (True, False):
        s = pkg.Simulation(p)
        if pin is not None:
            s.set_particles(pin)
        s.profile(profiled)
        rec = []
        for steps in (1, 2, 25, 30):
            s.step(steps)
            rec.append(s.series())
        assert s.kk == 58 and s.status() == 0
        runs.append({**read_all(s), "series": np.concatenate(rec)})
        s.close()
    assert_same(runs[1], runs[0], program)


SHAPES = [(64, 8, 1), (32, 8, 2), (64, 4, 4), (128, 2, 2)]


def batch_cases(cases, precision):
    """Programs of every boundary and rheology, with and without disks; the
    widths are a multiple of the batch tiles, one more and one less."""
    out = []
    for program, nx, ny, n, diam in (("c3", 128, 90, 12, 9.0), ("c6", 63, 120, 2, 10.0),
                                     ("c4", 64, 47, 1, 9.0), ("c1", 97, 61, 1, 8.0),
                                     ("c1", 40, 40, 0, 0.0)):
        p, pin = build(cases, program, nx, ny, n, diam, precision)
        p.series_every, p.series_capacity, p.series_particles = 3, 16, n
        out.append((p, turning(pin)))
    return out


def read_run(s):
    out = {"series": s.series(), "ux": s.field("ux"), "uy": s.field("uy"), "rho": s.field("rho")}
    if s.np:
        out["particles"] = s.particles()
    return out


def test_batch_kernels_and_single_runs_give_the_same_bits(pkg, cases):
    cs = batch_cases(cases, 1)
    want = []
    for p, pin in cs:
        s = pkg.Simulation(p)
        if pin is not None:
            s.set_particles(pin)
        s.step(40)
        want.append(read_run(s))
        s.close()
    for shape in SHAPES:
        b = pkg.Batch([p for p, _ in cs])
        b.set_tuning(*shape)
        for s, (_, pin) in zip(b.sims, cs):
            if pin is not None:
                s.set_particles(pin)
        b.step(40)
        for q, s in enumerate(b.sims):
            assert_same(read_run(s), want[q], (shape, q))
        b.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(64, 8, 1), (32, 8, 2)])
def test_batch_steps_between_a_simulations_own(pkg, cases, shape, precision):
    """A batch's simulation stepped on its own (the resident kernel: it swaps
    the disk state's copies, rotates the force accumulators and leaves the tile
    lists old) between steps of the batch."""
    cs = batch_cases(cases, precision)
    want = []
    for p, pin in cs:
        s = pkg.Simulation(p)
        if pin is not None:
            s.set_particles(pin)
        s.step(39)
        want.append(read_run(s))
        s.close()
    b = pkg.Batch([p for p, _ in cs])
    b.set_tuning(*shape)
    for s, (_, pin) in zip(b.sims, cs):
        if pin is not None:
            s.set_particles(pin)
    b.step(4)
    for s in b.sims:
        s.step(7)
    b.step(11)
    for q, s in enumerate(b.sims):  # odd and even, one launch and two, one step
        for n in ((5,), (2, 3), (4, 1), (1, 1, 3), (5,))[q]:
            s.step(n)
    b.step(12)
    for q, s in enumerate(b.sims):
        assert s.kk == 39 and s.status() == 0
        assert_same(read_run(s), want[q], (shape, q))
    b.close()
