"""The resident solve (csrc/cgres.cuh) gives the bits of the solve with a launch
per iteration: same arithmetic, same order of every sum, and quotients by a
corrected reciprocal that equal the divisions there. 120 iterations on
densities whose scales span 1e-9 to 1, which amplify a change of one rounding,
with loads and starting values on fixed DOFs as well. Equality is exact; what
each size ran is told by its number of launches.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.fem.solver import PCGSolver  # noqa: E402
from toptimization_b200.material import compute_Ke_2d, regularized_inverse  # noqa: E402

ITERS = 120
STEPS, COOPERATIVE = 1, 2
CLUSTER, COOP = 1, 2  # launches of a blocking resident solve


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("pre", ["none", "jacobi", "nodal_block_jacobi"])
@pytest.mark.parametrize("nx,ny,launches", [
    (3, 2, CLUSTER), (13, 13, CLUSTER), (97, 41, CLUSTER), (59, 100, CLUSTER),
    (1, 300, CLUSTER), (300, 1, COOP), (151, 49, COOP), (300, 170, COOP),
    (401, 310, COOP),  # the last CTA has empty groups
    (460, 270, COOP), (5, 17000, COOP),
    (420, 400, None)])  # beyond: a launch per iteration by itself
def test_same_bits_in_every_form(nx, ny, launches, pre, warm):
    rng = np.random.default_rng(nx + 3 * ny)
    Ke = compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    _lib.ensure_stiffness(Ke, inv, alpha)
    nn = (nx + 1) * (ny + 1)
    mask = np.zeros(nn, np.uint8)
    mask[:ny + 1] = 3
    mask[rng.integers(0, nn, 4)] = [1, 2, 3, 1]
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    rho = dev(10.0 ** rng.uniform(-3.0, 0.0, nx * ny))
    f, u0 = dev(rng.standard_normal(2 * nn)), dev(0.1 * rng.standard_normal(2 * nn))
    fixed = dev(mask)
    s = PCGSolver(nx, ny, 1e-9, 3.0, float(f @ f), preconditioner=pre, max_iter=ITERS, tol=1e-12)

    def solve(form):
        _lib.check(_lib.load().tpo_test_solve_form(form))
        u = u0.clone()
        info = s.solve(rho, f, fixed, u, warm_start=warm)
        _lib.check(_lib.load().tpo_test_solve_form(form))
        v, res = u0.clone(), s.result_buffer()
        s.solve_async(rho, f, fixed, v, res, warm_start=warm)
        torch.cuda.synchronize()
        late = PCGSolver.decode(res)
        assert torch.equal(u, v)
        assert (late.status, late.updates, late.rr) == (info.status, info.updates, info.rr)
        return u, info

    u, info = solve(0)
    ref, ref_info = solve(STEPS)
    if launches is None:
        assert info.launches == ref_info.launches
    else:
        assert info.launches == launches < ref_info.launches
    assert ref_info.launches > ref_info.updates > 0
    got = [(u, info)]
    if launches is not None:
        got.append(solve(COOPERATIVE))
        assert got[-1][1].launches == COOP
    for w, i in got:
        assert torch.isfinite(w).all()
        assert torch.equal(w, ref)
        assert (i.status, i.updates, i.rr) == (ref_info.status, ref_info.updates, ref_info.rr)
