"""The one-launch OC update against the oracle's bisection, at the sizes where
its forms change (one cluster, a cooperative grid with the elements held in
registers, one that streams them) and for every way its search can go: first
midpoint already a lower bound, first upper bound at the last midpoint, never
one, a move limit of zero, dc of either sign, non-finite dc, and dv given.

The candidate formula is evaluated at the midpoint the oracle stopped at, so
the densities differ by the rounding of one division, one square root and one
product: 4 ulp of a value below 1.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import simp64 as O  # noqa: E402
from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.optimizer import oc as OCm  # noqa: E402

TOL = 4 * 2.0 ** -53


def _steps(rho, dc, vf, move, dv):
    """The oracle's bisection, counting its steps."""
    lo, hi, steps = 0.0, 1e9, 0
    dv = np.ones_like(rho) if dv is None else dv
    while True:
        mid = 0.5 * (lo + hi)
        be = np.maximum(-dc / (mid * dv + 1e-20), 0.0)
        new = np.maximum(np.maximum(0.001, rho - move),
                         np.minimum(np.minimum(1.0, rho + move), rho * np.sqrt(be)))
        steps += 1
        if new.mean() > vf:
            lo = mid
        else:
            hi = mid
        if (hi - lo) / (hi + lo + 1e-30) < 1e-4 or steps >= 50:
            return mid, steps


def _run(rho, dc, vf, move=0.2, dv=None):
    n = rho.size
    g = _lib.grid(n, 1, 1e-9, 3.0)
    t = [torch.from_numpy(a).cuda() if a is not None else None for a in (rho, dc, dv)]
    out = torch.empty_like(t[0])
    res = torch.empty(4, dtype=torch.float64, device="cuda")
    OCm.oc_update(g, vf, move, t[0], t[1], out, res, OCm.oc_workspace(g, "cuda"), dv=t[2])
    with np.errstate(all="ignore"):
        ref, change = O.oc_update(rho, dc, vf, move, dv)
        mid, steps = _steps(rho, dc, vf, move, dv)
    got, r = out.cpu().numpy(), res.cpu().numpy()
    assert np.abs(got - ref).max() <= TOL
    assert abs(r[0] - change) <= TOL
    assert r[1] == pytest.approx(ref.mean(), rel=1e-12)
    assert r[2] == mid and r[3] == steps


@pytest.mark.parametrize("n", [1, 5, 1023, 1025, 16384, 16385, 150001, 303104, 303105, 700003])
@pytest.mark.parametrize("with_dv", [False, True])
def test_sizes(n, with_dv):
    rng = np.random.default_rng(n)
    rho = rng.uniform(0.001, 1.0, n)
    dc = -rng.exponential(1.0, n) * 10.0 ** rng.uniform(-6, 2, n)
    _run(rho, dc, 0.4, dv=rng.uniform(0.5, 2.0, n) if with_dv else None)


@pytest.mark.parametrize("scale", [1e18, 1e9, 1e-3, 1e-9, 1e-14, 1e-30])
def test_search_ranges(scale):
    """Multipliers from above the first midpoint to below the last."""
    rng = np.random.default_rng(3)
    rho = rng.uniform(0.1, 0.9, 4000)
    _run(rho, -scale * rng.uniform(0.5, 2.0, 4000), 0.45)


@pytest.mark.parametrize("vf", [0.0005, 0.999, 1.5])
def test_targets_out_of_reach(vf):
    rng = np.random.default_rng(4)
    _run(rng.uniform(0.3, 0.6, 3000), -rng.exponential(1.0, 3000), vf)


def test_odd_values():
    rng = np.random.default_rng(5)
    rho = rng.uniform(0.05, 1.0, 20000)
    dc = rng.standard_normal(20000)  # either sign
    dc[::17] = 0.0
    dc[5], dc[6] = -np.inf, np.inf
    _run(rho, dc, 0.3)
    _run(rho, -np.abs(dc), 0.3, move=0.05)


@pytest.mark.parametrize("n", [64, 32768, 524288])
def test_lowest_midpoints_count_the_regulariser(n):
    """At the 49th midpoint, 1e9 / 2^49, the reference's 1e-20 beside lambda
    lowers a candidate by 2.8e-15, about 13 ulp. The target lies half-way
    between the volumes with and without it (equal elements, a power of two of
    them: their mean is the candidate); the kernel's own rounding is below 4 ulp."""
    lam = 1e9 / 2.0 ** 49
    with_, without = 0.5 * np.sqrt(lam / (lam + 1e-20)), 0.5
    assert 5e-16 < without - with_ < 2e-15
    _run(np.full(n, 0.5), np.full(n, -lam), 0.5 * (with_ + without))


@pytest.mark.parametrize("n", [4 * 148 * 1024, 4 * 148 * 1024 + 1])
@pytest.mark.parametrize("either_sign", [False, True])
def test_two_levels_per_pass(n, either_sign):
    """dv on either side of the size from which a pass takes two levels of the
    bisection instead of three (148 SMs). The volumes' rounding, below 1e-12 of
    them, is far from the target at every midpoint but the last few, whose
    lambda then differ by 1e-4 at most; the seeds below do not meet that."""
    rng = np.random.default_rng(6)
    rho = rng.uniform(0.001, 1.0, n)
    dc = -rng.exponential(1.0, n)
    dv = rng.uniform(-0.5 if either_sign else 0.5, 2.0, n)
    _run(rho, dc, 0.4, dv=dv)
