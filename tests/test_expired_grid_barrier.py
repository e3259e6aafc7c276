"""A grid barrier that expires (k_steps, k_adj_levels) must not leave the
launches queued behind it spinning: the host has counted their arrivals
already, so the count stays short for all of them.  lbm_selftest_wait makes a
barrier wait run out with a small limit and queues a multi-step launch behind
it, which has to return without a step; nothing here faults or hangs a GPU."""

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LBM_E_TIMEOUT = -6


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("warm", [0, 1, 7])
def test_launch_behind_an_expired_barrier_does_nothing(pkg, cases, precision, warm):
    p, pin = cases.shipped_c6(60, 120)
    p.precision = precision
    p.series_every = 0
    sim = pkg.Simulation(p)
    sim.set_particles(pin)
    if warm:
        sim.step(warm)
    before = sim.particles()
    assert sim.status() == 0
    t0 = time.perf_counter()
    sim.selftest_wait(256)  # LbmError(LBM_E_STATE) if the launch behind it stepped
    assert time.perf_counter() - t0 < 1.0  # 2^22 polls take several seconds
    assert sim.status() == LBM_E_TIMEOUT and sim.kk == warm
    with pytest.raises(pkg.LbmError) as err:
        sim.particles()
    assert err.value.code == LBM_E_TIMEOUT
    with pytest.raises(pkg.LbmError):
        sim.adjoint(1, 2)
    sim.close()
    # the device and other handles go on
    ref, again = [], pkg.Simulation(p)
    again.set_particles(pin)
    if warm:
        again.step(warm)
    ref = again.particles()
    assert again.status() == 0 and np.array_equal(ref, before)
    again.close()
