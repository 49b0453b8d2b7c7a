"""libtpo's host code on a machine of two devices: launch attributes belong to
the device that was current when they were set, so every device a process uses
needs its own, and a device that cannot give the resident solve what it needs
still solves. On a CUDA runtime over host memory (conftest.host_lib).
"""

import ctypes

import numpy as np
import pytest

from conftest import host_launches
from toptimization_b200 import _lib

OPT_IN = 227 * 1024


def _on(L, dev):
    assert L.fake_set_device(dev) == 0
    from toptimization_b200.material import compute_Ke_2d, regularized_inverse
    Ke = compute_Ke_2d(1.0, 0.3)
    inv, alpha = regularized_inverse(Ke)
    as_pd = lambda a: np.ascontiguousarray(a).ctypes.data_as(_lib._PD)  # noqa: E731
    assert L.tpo_set_stiffness(as_pd(Ke), as_pd(inv), alpha) == 0


def _aligned(nbytes):
    raw = np.zeros(nbytes + 256, np.uint8)
    at = -raw.ctypes.data % 256
    return raw[at:at + nbytes]


def _solve(L, nx, ny, pre="jacobi", asynchronous=False, precision=0, recurrence=0):
    """The solve's return code and its launches, one dict each."""
    g = _lib.grid(nx, ny, 1e-9, 3.0)
    c = _lib.TpoSolveCfg(precond=_lib.PRECOND[pre], precision=precision, max_iter=3, tol=1e-8,
                         f_norm_sq=1.0, inner_tol=1e-3, max_outer=4, poll_every=16,
                         recurrence=recurrence)
    nn = (nx + 1) * (ny + 1)
    rho, f, u = _aligned(8 * nx * ny), _aligned(16 * nn), _aligned(16 * nn)
    fixed, out = _aligned(nn), _aligned(256)
    ws = _aligned(L.tpo_pcg_workspace_bytes(g, c))
    L.fake_log()
    p = lambda a: a.ctypes.data  # noqa: E731
    if asynchronous:
        rc = L.tpo_pcg_solve_async(g, c, p(rho), p(f), p(fixed), p(u), p(ws), ws.size, p(out), None)
    else:
        res = _lib.TpoSolveResult()
        rc = L.tpo_pcg_solve(g, c, p(rho), p(f), p(fixed), p(u), p(ws), ws.size,
                             ctypes.byref(res), None)
    return rc, host_launches(L)


def _named(launches, kernel):
    return [x for x in launches if x["name"].startswith(kernel + "<")]


# one cluster of up to 8 CTAs, of up to 16, cooperative with little and with
# much shared memory, three groups of 480 threads; the first grid beyond
SIZES = [(13, 13), (97, 41), (151, 49), (400, 200), (460, 270), (900, 900)]


@pytest.mark.parametrize("asynchronous", [False, True])
@pytest.mark.parametrize("pre", ["none", "jacobi", "nodal_block_jacobi"])
def test_every_device_of_a_process_solves(host_lib, pre, asynchronous):
    for nx, ny in SIZES:
        seen = []
        for dev in (0, 1, 0):
            _on(host_lib, dev)
            rc, launches = _solve(host_lib, nx, ny, pre, asynchronous)
            assert rc == 0, host_lib.tpo_last_error_string()
            assert launches and all(x["dev"] == dev and x["err"] == 0 for x in launches)
            assert bool(_named(launches, "k_cgres")) == (nx * ny < 500_000)
            seen.append([{k: v for k, v in x.items() if k != "dev"} for x in launches])
        assert seen[0] == seen[1] == seen[2]


def test_cluster_size_is_each_devices_own(host_lib):
    host_lib.fake_limits(1, 8, OPT_IN)  # no room for 16 CTAs in a cluster of device 1
    for dev, most in ((0, 16), (1, 8), (0, 16)):
        _on(host_lib, dev)
        sizes = []
        for nx, ny in SIZES[:-1]:
            rc, launches = _solve(host_lib, nx, ny)
            assert rc == 0, host_lib.tpo_last_error_string()
            (k,) = _named(launches, "k_cgres")
            assert k["err"] == 0
            sizes.append(k["cluster"])
        assert max(sizes) > 8 if most == 16 else 1 < max(sizes) <= 8


def test_device_without_the_shared_memory_solves_with_a_launch_per_iteration(host_lib):
    host_lib.fake_limits(1, 16, 48 * 1024)
    for dev, resident in ((1, False), (0, True), (1, False)):
        _on(host_lib, dev)
        for nx, ny in SIZES[:-1]:
            rc, launches = _solve(host_lib, nx, ny)
            assert rc == 0, host_lib.tpo_last_error_string()
            assert all(x["err"] == 0 for x in launches)
            assert bool(_named(launches, "k_cgres")) == resident
            assert bool(_named(launches, "k_cgstep")) != resident


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("pre", list(_lib.PRECOND))
def test_two_launch_forms_on_every_device(host_lib, pre, precision):
    for dev in (0, 1):
        _on(host_lib, dev)
        for asynchronous in (False, True):
            rc, launches = _solve(host_lib, 400, 200, pre, asynchronous, precision, recurrence=1)
            assert rc == 0, host_lib.tpo_last_error_string()
            assert launches and all(x["dev"] == dev and x["err"] == 0 for x in launches)
            assert not _named(launches, "k_cgres") and not _named(launches, "k_cgstep")
