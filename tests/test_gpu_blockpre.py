"""The element-block preconditioner's kernel (tiles of 30 rows x 16 columns)
against the oracle's PCG at the edges of its tiles and of the groups of four
tiles whose sums are added together; FP64 and mixed storage, zero and warm
start.

Eight iterations with densities in [0.3, 1]: rounding errors of a few hundred
ulp at most, 1e-11 of the solution; with FP32-stored vectors the same in units
of 2^-24: a few hundred roundings, 2e-5.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import simp64 as O  # noqa: E402
from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.fem.solver import PCGSolver  # noqa: E402
from toptimization_b200.material import compute_Ke_2d, regularized_inverse  # noqa: E402


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-5)])
@pytest.mark.parametrize("nx,ny", [(2, 2), (15, 29), (16, 30), (17, 31), (3, 119), (47, 120),
                                   (130, 5), (64, 150)])
def test_matches_oracle(nx, ny, precision, tol):
    rng = np.random.default_rng(nx * 1000 + ny)
    Ke = compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    _lib.ensure_stiffness(Ke, inv, alpha)
    mesh = O.Mesh2D(nx, ny, Ke, np.arange(2 * (ny + 1)))
    f = rng.standard_normal(mesh.n_dofs)
    f[mesh.is_fixed] = 0.0
    mask = np.zeros(mesh.n_nodes, np.uint8)
    mask[:ny + 1] = 3
    rho = rng.uniform(0.3, 1.0, nx * ny)
    u0 = 0.1 * rng.standard_normal(mesh.n_dofs)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    iters = 8 if nx > 2 else 4
    s = PCGSolver(nx, ny, 1e-9, 3.0, float(f @ f), preconditioner="block_jacobi",
                  precision=precision, max_iter=iters, tol=1e-30)
    scale = O.simp_scale(rho, 1e-9, 3.0)
    for warm in (False, True):
        start = np.where(mesh.is_fixed, 0.0, u0) if warm else np.zeros(mesh.n_dofs)
        ref = O.pcg(mesh, scale, f, start, 1e-30, iters, "block_jacobi")
        u = dev(u0.copy())
        info = s.solve(dev(rho), dev(f), dev(mask), u, warm_start=warm)
        assert info.updates == ref.iters
        assert np.linalg.norm(u.cpu().numpy() - ref.u) <= tol * np.linalg.norm(ref.u)
