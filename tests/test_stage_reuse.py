"""FP64 step kernels that put a node's populations back into their TMA stage
while they visit the disks (lbm_lattice.cuh, node_force): the stage is then
refilled by TMA, so every block here works through several tiles with disks
per stage.  The one-node-per-thread batch kernel stages nothing; it shares
the node arithmetic, so the results are the same to the bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(cases, program, nx, ny):
    if program == "c3":
        p = cases.shipped_c3(nx, ny)
        p.gravity = -5e-5
        p.rep_zeta = 2.0
    else:  # Bingham: 512-node tiles with an omega box
        p, _ = cases.shipped_c6(nx, ny)
        p.contact_test = 0
    p.precision = 0
    p.series_every = 0
    return p


def disks(cases, nx, ny, diam, pitch):
    """A grid of disks over the whole lattice, each moving and turning."""
    x, y = np.meshgrid(np.arange(pitch, nx - pitch, pitch, dtype=float),
                       np.arange(pitch, ny - pitch, pitch, dtype=float))
    k = np.arange(x.size)
    uvw = np.stack([1e-3 * ((k % 3) - 1), 1e-3 * ((k % 4) - 1.5), 1e-4 * ((k % 5) - 2)], axis=1)
    return cases.pin_array(np.stack([x.ravel() + 0.3, y.ravel() - 0.2], axis=1), diam,
                           1.2 + 0.01 * (k % 7), uvw=uvw)


def read(s):
    return {"particles": s.particles(), "ux": s.field("ux"), "uy": s.field("uy"),
            "rho": s.field("rho")}


# (1023, 767): 3072 tiles of 256 nodes or 1536 of 512 over at most 294 blocks;
# (1024, 515): the wall column in tiles of its own, a ragged last row of tiles
@pytest.mark.parametrize("program", ["c3", "c6"])
@pytest.mark.parametrize("nx,ny", [(1023, 767), (1024, 515)])
def test_stages_with_disks_are_refilled_in_order(pkg, cases, program, nx, ny):
    p = params(cases, program, nx, ny)
    pin = disks(cases, nx, ny, 10.0, 24.0)
    steps = 24
    s = pkg.Simulation(p)
    s.set_particles(pin)
    s.step(steps)
    assert s.status() == 0
    got = {"single": read(s)}
    s.close()
    for name, shape in (("staged batch", (64, 8, 1)), ("unstaged batch", (32, 8, 4))):
        b = pkg.Batch([p, p])
        b.set_tuning(*shape)
        for q in b.sims:
            q.set_particles(pin)
        b.step(steps)
        got[name] = read(b.sims[1])
        b.close()
    want = got["unstaged batch"]
    for name in ("single", "staged batch"):
        for k, w in want.items():
            assert np.array_equal(got[name][k], w), (name, k)
