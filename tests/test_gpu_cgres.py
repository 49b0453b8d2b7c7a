"""The resident solve (one cooperative launch, cgres.cuh) against the oracle's
PCG: grids of one tile, of many, thin ones, ones whose sizes leave ragged last
tiles, the largest that fit and the first that does not; every point
preconditioner, zero and warm start.

Twelve iterations from the same start with densities in [0.3, 1]: both sides
carry rounding errors of a few hundred ulp at most (tens of operations per
value and iteration, no amplification this early), 1e-11 of the solution.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import simp64 as O  # noqa: E402
from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.fem.solver import PCGSolver  # noqa: E402
from toptimization_b200.material import compute_Ke_2d, regularized_inverse  # noqa: E402

TOL = 1e-11


def _case(nx, ny, seed):
    rng = np.random.default_rng(seed)
    Ke = compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    _lib.ensure_stiffness(Ke, inv, alpha)
    some = rng.integers(0, 2 * (nx + 1) * (ny + 1), 5 if nx * ny > 20 else 0)
    fixed = np.unique(np.r_[np.arange(2 * (ny + 1)), some])  # left edge, some single DOFs
    mesh = O.Mesh2D(nx, ny, Ke, fixed)
    f = rng.standard_normal(mesh.n_dofs)
    f[mesh.is_fixed] = 0.0
    mask = np.zeros(mesh.n_nodes, np.uint8)
    for d in fixed:
        mask[d // 2] |= 1 << (d % 2)
    return mesh, f, mask, rng.uniform(0.3, 1.0, nx * ny), 0.1 * rng.standard_normal(mesh.n_dofs)


@pytest.mark.parametrize("pre", ["none", "jacobi", "nodal_block_jacobi"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 300), (300, 1), (13, 13), (14, 14), (29, 61),
                                   (97, 41), (333, 170), (401, 310), (370, 390)])
def test_matches_oracle(nx, ny, pre):
    mesh, f, mask, rho, u0 = _case(nx, ny, nx + 7 * ny)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    iters = 12 if nx * ny > 1 else 3  # one element: four free DOFs
    s = PCGSolver(nx, ny, 1e-9, 3.0, float(f @ f), preconditioner=pre, max_iter=iters, tol=1e-30)
    scale = O.simp_scale(rho, 1e-9, 3.0)
    for warm in (False, True):
        start = np.where(mesh.is_fixed, 0.0, u0) if warm else np.zeros(mesh.n_dofs)
        ref = O.pcg(mesh, scale, f, start, 1e-30, iters, pre)
        u = dev(u0.copy())
        info = s.solve(dev(rho), dev(f), dev(mask), u, warm_start=warm)
        got = u.cpu().numpy()
        assert info.updates == ref.iters
        assert np.linalg.norm(got - ref.u) <= TOL * np.linalg.norm(ref.u)
        res = s.result_buffer()
        v = dev(u0.copy())
        s.solve_async(dev(rho), dev(f), dev(mask), v, res, warm_start=warm)
        torch.cuda.synchronize()
        assert torch.equal(u, v) and PCGSolver.decode(res).updates == info.updates
