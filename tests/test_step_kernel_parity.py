"""The particle and step kernels on the small lattices of the parity tests.

lbm_step takes the resident kernel there; a handle being profiled (lbm_profile)
takes one launch per kernel.  The oracle and golden parity tests of
test_gpu_parity run here once more with every handle profiled, so that each
boundary, rheology and precision is also compared through the step kernel's
tiles.  Then lattices whose wall column NX starts a step-kernel tile of its
own, ends one or lies inside one (tiles are 64 nodes wide in FP64 and 128 in
FP32), with a disk whose PHI ring reaches the column: the step kernel gives
the resident kernel's bits and, in FP64, the oracle's results."""

import importlib
import types

import numpy as np
import pytest

import test_gpu_parity as parity
from oracle.oracle import Oracle
from test_gpu_parity import (  # noqa: F401 - collected here, with this file's pkg
    test_c1_matches_reference_golden, test_c1_nonnewtonian_strain_feq_fp64,
    test_c1_offcentre_rotation_fp64, test_c1_zouhe_fp64,
    test_c2_two_disks_match_reference_golden,
    test_c4_oscillating_cylinder_matches_reference_golden, test_c6_bingham_fp64,
    test_c3_casson_fp64, test_fp32_shifted_vs_fp64_oracle, test_multiparticle_fp64,
    test_series_and_mean_density_fp64, test_wall_column_pass)

pytestmark = pytest.mark.gpu


@pytest.fixture
def plain():
    """The package as the other tests have it."""
    return importlib.import_module("2d_nnf_lbm_b200")


@pytest.fixture
def cases(plain):
    return plain.cases


@pytest.fixture
def pkg(plain):
    """The package with every handle profiled from its start."""

    class Profiled(plain.Simulation):
        def __init__(self, *args, **kw):
            super().__init__(*args, **kw)
            self.profile(True)

    return types.SimpleNamespace(**{**vars(plain), "Simulation": Profiled})


COLUMNS = [("c3", nx, ny) for nx in (63, 64, 65, 127, 128, 129) for ny in (47, 48)]
COLUMNS += [("c6", nx, ny) for nx in (63, 64, 127, 128, 129) for ny in (48, 55)]


def column_case(cases, program, nx, ny, precision):
    if program == "c3":
        p = cases.shipped_c3(nx, ny)
        p.gravity = -5e-5
    else:  # Bingham: 512-node tiles with an omega box
        p, _ = cases.shipped_c6(nx, ny)
        p.record_stress = 1
    p.precision = precision
    p.wall_model = 2  # no wall repulsion: the disk stays on the wall column
    p.contact_test = 0
    p.series_every, p.series_capacity, p.series_particles = 4, 8, 2
    pin = cases.pin_array([[nx - 5.2, 30.0], [12.4, 14.7]], 10.0, [1.5, 1.3],
                          uvw=[[0.0, 0.0, 2e-3], [1e-3, 0.0, -1e-3]])
    return p, pin


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("program,nx,ny", COLUMNS)
def test_disk_on_the_wall_column(plain, pkg, cases, program, nx, ny, precision):
    p, pin = column_case(cases, program, nx, ny, precision)
    got = []
    for lib in (pkg, plain):
        s = lib.Simulation(p)
        s.set_particles(pin)
        s.step(30)
        s.step(10)
        assert s.kk == 40 and s.status() == 0
        f, om, ps = s.get_state()
        out = {"f": f, "omega": om, "state": ps, "series": s.series()}
        out.update({k: s.field(k) for k in ("ux", "uy", "rho", "phi", "gx", "gy")})
        if p.record_stress:
            out["tau12"] = s.field("tau12")
        got.append((out, s))
    for k, w in got[1][0].items():
        assert np.array_equal(got[0][0][k], w, equal_nan=True), k
    assert got[0][0]["phi"][:, nx].max() > 0.0
    if precision == 0:
        ref = Oracle(p)
        ref.set_particles(pin)
        ref.step(40)
        # Bingham: m = 5.5e6 amplifies ulp-level differences (test_c6_bingham_fp64)
        parity.compare_all(got[0][1], ref, rtol=1e-8 if p.rheology else parity.RTOL64)
    for _, s in got:
        s.close()
