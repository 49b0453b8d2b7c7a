"""Launch shapes that a kernel's speed rests on, from the host code alone (on a CUDA
runtime over host memory, conftest.host_lib)."""

import numpy as np
import pytest

from conftest import host_launches
from toptimization_b200 import _lib


@pytest.mark.parametrize("sens", [False, True])
@pytest.mark.parametrize("rmin", [8.2, 9.0, 12.5, 16.0])
def test_large_filter_radii_have_256_threads_per_tile(host_lib, rmin, sens):
    """Beyond the register form a tile's shared memory, 21 to 41 KB, limits the CTAs
    of an SM, so the threads of a CTA are the warps that hide its loads."""
    nx, ny = 70, 41
    a = [np.zeros(nx * ny) for _ in range(3)]
    p = [x.ctypes.data for x in a]
    g = _lib.grid(nx, ny, 1e-9, 3.0)
    if sens:
        rc = host_lib.tpo_sensitivity_filter(g, rmin, p[0], p[1], p[2], None)
    else:
        rc = host_lib.tpo_density_filter(g, rmin, p[0], p[1], None, None, None)
    assert rc == 0, host_lib.tpo_last_error_string()
    (k,) = host_launches(host_lib)
    assert k["err"] == 0 and k["threads"] == 256 and k["grid"] == 3 * 2


@pytest.mark.parametrize("rmin,kernel", [(0.9, "taps<0,27>"), (1.0, "taps<0,27>"),
                                         (2.0, "taps<0,27>"), (2.1, "taps<0,304>"),
                                         (4.1, "taps<0,304>"), (4.4, "filter<0>")])
def test_filter3_argument_no_larger_than_its_list(host_lib, rmin, kernel):
    """A neighbour list is a kernel argument; a long one delays the launch."""
    n = 9 * 8 * 7
    a = [np.zeros(n) for _ in range(2)]
    g = _lib.grid3(9, 8, 7, 1e-9, 3.0)
    rc = host_lib.tpo3_density_filter(g, rmin, a[0].ctypes.data, a[1].ctypes.data, None)
    assert rc == 0, host_lib.tpo_last_error_string()
    (k,) = host_launches(host_lib)
    assert k["err"] == 0 and k["name"].endswith(kernel), k["name"]
