"""Buffers that lbm_adjoint keeps on the handle, across gradients of different
sizes: one without levels (n1 = 1) needs no checkpoints, and a change of the
disk count replaces the per-disk buffers."""

import numpy as np
import pytest

from test_steps_resident import build

pytestmark = pytest.mark.gpu


def test_gradient_without_levels_after_one_with(pkg, cases):
    """The checkpoints are released once: a handle created in between may hold
    memory at their old address when the first handle is closed."""
    p, few = build(cases, "c3", 95, 130, 2, 8.0, 0)
    p.contact_test, p.series_every = 0, 0
    _, many = build(cases, "c3", 95, 130, 40, 8.0, 0)
    s = pkg.Simulation(p)
    start = s.get_state()
    s.set_particles(few)
    s.adjoint(10, 12)
    s.set_state(0, *start[:2], np.zeros((0, 20)))
    s.set_particles(many)
    s.adjoint(1, 1)
    others = []
    for _ in range(3):
        o = pkg.Simulation(p)
        o.set_particles(few)
        o.step(20)
        others.append((o, o.particles(), o.field("ux")))
    s.close()
    more = [pkg.Simulation(p) for _ in range(3)]  # would take what is free
    for o, parts, ux in others:
        assert np.array_equal(o.particles(), parts) and np.array_equal(o.field("ux"), ux)
        assert o.status() == 0
        o.close()
    for m in more:
        m.close()


def test_refused_allocation_leaves_no_error_behind(pkg, cases):
    """A gradient that does not fit in memory is LBM_E_NOMEM, and the calls
    after it are not."""
    torch = pytest.importorskip("torch")
    p, pin = build(cases, "c6", 280, 280, 2, 20.0, 0)
    p.contact_test, p.series_every = 0, 0
    s = pkg.Simulation(p)
    s.set_particles(pin)
    before = s.particles()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(pkg.LbmError) as err:
            s.adjoint(400, 404, checkpoint_every=200)
        assert err.value.code == -3  # LBM_E_NOMEM
        assert np.array_equal(s.particles(), before)
        assert np.isfinite(s.field("ux")).all() and s.status() == 0
    finally:
        del taken
        torch.cuda.empty_cache()
    s.step(10)
    assert s.status() == 0 and s.kk == 10
    s.close()
