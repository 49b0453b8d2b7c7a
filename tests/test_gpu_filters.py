"""The filters and sensitivities at the places where their kernels change:
every radius of the register form and the first beyond it, tiles with
remainders, grids smaller than the box, 3D neighbour lists up to their limit
and the box walk beyond it; non-finite values only where a positive weight
reaches; the 3D energy from the element's modes against extended precision.

Filter tolerance: numerator and denominator are sums of at most 800 positive
products, in any order within 800 ulp of the exact ones: 2e-13 relative. (The
sums of the tests are far shorter than that on average; the oracle's own are
as long.)
"""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import simp64 as O  # noqa: E402
from toptimization_b200 import _lib  # noqa: E402
from toptimization_b200.fem import kernels as K  # noqa: E402
from toptimization_b200.material import compute_Ke_3d, regularized_inverse  # noqa: E402
from toptimization_b200.optimizer import filter as F  # noqa: E402

TOL = 2e-13


def _check(g, shape, rmin, nz=0):
    rng = np.random.default_rng(int(10 * rmin) + shape[0])
    n = int(np.prod(shape))
    x, rho = rng.uniform(0.1, 1.0, n), rng.uniform(0.1, 1.0, n)
    H, Hs = O.filter_matrix(shape[0], shape[1], rmin, nz)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    F.density_filter(g, rmin, dev(x), out)
    assert np.abs(out.cpu().numpy() / O.density_filter(H, Hs, x) - 1).max() < TOL
    F.sensitivity_filter(g, rmin, dev(rho), dev(x), out)
    ref = (H @ (rho * x)) / (rho * np.asarray(Hs).reshape(-1) + 1e-20)
    assert np.abs(out.cpu().numpy() / ref - 1).max() < TOL


@pytest.mark.parametrize("rmin", [0.6, 1.0, 1.5, 2.0, 2.5, 3.3, 4.0, 4.6, 5.9, 6.2, 7.0, 8.0, 8.3])
@pytest.mark.parametrize("nx,ny", [(1, 5), (3, 2), (33, 32), (40, 31), (65, 97)])
def test_filter2(nx, ny, rmin):
    _check(_lib.grid(nx, ny, 1e-9, 3.0), (nx, ny), rmin)


@pytest.mark.parametrize("rmin", [0.7, 1.0, 1.5, 2.2, 3.1, 4.1, 4.4, 6.5])
@pytest.mark.parametrize("shape", [(1, 1, 9), (5, 4, 3), (17, 9, 12)])
def test_filter3(shape, rmin):
    _check(_lib.grid3(*shape, 1e-9, 3.0), shape, rmin, shape[2])


@pytest.mark.parametrize("nz", [0, 7])
def test_infinite_value_spreads_only_under_positive_weights(nz):
    shape = (20, 37) if not nz else (11, 9, nz)
    g = _lib.grid3(*shape, 1e-9, 3.0) if nz else _lib.grid(*shape, 1e-9, 3.0)
    rmin, at = 2.5, tuple(s // 2 for s in shape)
    x = np.ones(shape)
    x[at] = np.inf
    out = torch.empty(x.size, dtype=torch.float64, device="cuda")
    F.density_filter(g, rmin, torch.from_numpy(x.reshape(-1)).cuda(), out)
    dist = np.sqrt(sum((np.arange(s).reshape([-1 if i == d else 1 for i in range(len(shape))])
                        - at[d]) ** 2 for d, s in enumerate(shape)))
    assert np.array_equal(np.isinf(out.cpu().numpy().reshape(shape)), dist < rmin)
    assert not np.isnan(out.cpu().numpy()).any()


def test_energy3_from_modes_is_no_less_exact():
    """uKu of a smooth displacement with a large rigid part cancels; against
    extended precision the modal form has to be at least as close as the dense
    product in 64 bits."""
    n = (9, 7, 8)
    Ke = compute_Ke_3d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    _lib.ensure_stiffness3(Ke, inv, alpha)
    rng = np.random.default_rng(2)
    mesh = O.Mesh3D(*n, Ke, np.array([0]))
    X = np.meshgrid(*[np.arange(k + 1) / k for k in n], indexing="ij")
    u = np.stack([40.0 + 3.0 * math.pi * X[0] ** 2 + np.sin(2.0 * X[1] + d) + 0.1 * X[2] * X[0]
                  for d in range(3)], axis=-1).reshape(-1)
    rho = rng.uniform(0.1, 1.0, mesh.n_elem)
    ue = u[mesh.edof].astype(np.longdouble)
    uku = np.einsum("ei,ij,ej->e", ue, Ke.astype(np.longdouble), ue)
    exact = -3 * rho.astype(np.longdouble) ** 2 * (1 - np.longdouble(1e-9)) * uku
    dense, _ = O.sensitivity(mesh, u, rho, 1e-9, 3.0)
    g = _lib.grid3(*n, 1e-9, 3.0)
    dc = torch.empty(mesh.n_elem, dtype=torch.float64, device="cuda")
    c = torch.empty(1, dtype=torch.float64, device="cuda")
    K.sensitivity(g, torch.from_numpy(rho).cuda(), torch.from_numpy(u).cuda(), dc, c,
                  K.sensitivity_workspace(g, "cuda"))
    err = lambda v: float(np.linalg.norm((v - exact).astype(float)))  # noqa: E731
    assert err(dc.cpu().numpy()) <= err(dense)
