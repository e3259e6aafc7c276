"""The checked build over every route (tests/checked_routes.py): the cases run
once on the ordinary library and once on the checked one (a child process), no
check may fire and the results must be the same -- bit for bit (both builds
round alike, FP32 included), the gradients within 1e-12 (FP64) and 1e-5
(FP32) of each entry's kind: their per-disk sums are FP64 atomics in no fixed
order, of FP32 terms that cancel."""

import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)
import checked_routes  # noqa: E402


@pytest.mark.parametrize("name", ["lbm_steps.cuh", "lbm_adjoint.cu", "lbm_lattice.cuh",
                                  "lbm_particles.cu"])
def test_every_kernel_of_a_step_carries_index_checks(pkg, name):
    """The checks are written at the accesses: a kernel without any is not
    checked, however green the run below is."""
    path = os.path.join(os.path.dirname(pkg.__file__), "csrc", name)
    with open(path) as fh:
        assert "LBM_IN(" in fh.read()


@pytest.mark.gpu
def test_checked_build_over_every_route(pkg, tmp_path):
    want = checked_routes.run_cases(pkg)
    assert int(want["checked_build"]) == 0
    out = str(tmp_path / "checked.npz")
    env = dict(os.environ)
    env["LBM2D_LIBRARY"] = os.path.join(os.path.dirname(pkg.library_path()), "liblbm2d_checked.so")
    r = subprocess.run([sys.executable, os.path.join(HERE, "checked_routes.py"), out], env=env,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    got = dict(np.load(out))
    assert int(got["checked_build"]) == 1
    assert set(got) == set(want)
    for k, v in got.items():
        w = want[k]
        if k == "checked_build":
            continue
        if k.endswith("status"):
            assert int(v) == 0, (k, int(v))  # 0: no LBM_E_BOUNDS, no other error
        elif k.endswith("_grad"):
            fp64 = "0" in k.split("_")[0 if k.startswith("res") else 1]
            n = (len(w) - 2) // 3
            for kind in (slice(0, 1), slice(1, 2), slice(2, 2 + n), slice(2 + n, None)):
                tol = (1e-12 if fp64 else 1e-5) * np.max(np.abs(w[kind]))
                assert np.all(np.abs(v[kind] - w[kind]) <= tol), (k, kind, v[kind], w[kind])
        else:
            assert np.array_equal(v, w, equal_nan=True), k
