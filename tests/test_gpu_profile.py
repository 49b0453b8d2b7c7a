"""tpo_profile's byte counts: a solve that keeps its vectors on the chip counts the
caller's arrays once, whatever its iterations; one with a launch per iteration
counts the vectors of every launch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.fem.solver import PCGSolver  # noqa: E402
from toptimization_b200.material import compute_Ke_2d, regularized_inverse  # noqa: E402


def _profile(nx, ny, iters, warm):
    rng = np.random.default_rng(1)
    Ke = compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    _lib.ensure_stiffness(Ke, inv, alpha)
    nn = (nx + 1) * (ny + 1)
    mask = np.zeros(nn, np.uint8)
    mask[:ny + 1] = 3
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    f = rng.standard_normal(2 * nn)
    s = PCGSolver(nx, ny, 1e-9, 3.0, float(f @ f), preconditioner="jacobi", max_iter=iters, tol=1e-30)
    args = dev(rng.uniform(0.3, 1.0, nx * ny)), dev(f), dev(mask), dev(np.zeros(2 * nn))
    _lib.check(_lib.load().tpo_profile_enable(1))
    _lib.check(_lib.load().tpo_profile_reset())
    s.solve(*args, warm_start=warm)
    p = _lib.profile_read()
    _lib.check(_lib.load().tpo_profile_enable(0))
    assert p["step_launches"] == iters and p["step_ms"] > 0.0
    return p["step_bytes"]


@pytest.mark.parametrize("nx,ny", [(97, 41), (300, 170)])  # cluster, cooperative
def test_resident_solve(nx, ny):
    nn = (nx + 1) * (ny + 1)
    once = 8 * nx * ny + 16 * nn + nn + 16 * nn  # rho, f, mask; u
    for iters in (5, 40):
        assert _profile(nx, ny, iters, False) == once
        assert _profile(nx, ny, iters, True) == once + 16 * nn


def test_launch_per_iteration():
    nx, ny = 700, 500
    nn = (nx + 1) * (ny + 1)
    per = 9 * 16 * nn + 8 * nx * ny + nn  # r, w, s, p in and out, x every second time; scales, mask
    assert _profile(nx, ny, 6, False) == 6 * per
