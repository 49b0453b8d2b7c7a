import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parent.parent
GOLDEN = REPO / "tests" / "golden"
if str(REPO) not in sys.path:
    sys.path.insert(0, str(REPO))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and libtpo")


def pytest_collection_modifyitems(config, items):
    try:
        import torch
        have_cuda = torch.cuda.is_available()
    except Exception:  # pragma: no cover
        have_cuda = False
    if have_cuda:
        return
    skip = pytest.mark.skip(reason="no CUDA device in this environment")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


def golden(name: str):
    return np.load(GOLDEN / f"{name}.npz")


@pytest.fixture(scope="session")
def tpo_built():
    """Build libtpo if stale (the GPU machines carry the prebuilt .so)."""
    from toptimization_b200.csrc import build
    build.build()
    from toptimization_b200 import _lib
    return _lib.load()


@pytest.fixture(scope="session")
def host_build(tmp_path_factory):
    """libtpo's host code over a CUDA runtime in host memory (fake_cuda/runtime.cpp)
    that checks each launch and logs it. Nothing runs: the device code stays
    text, unoptimised."""
    from toptimization_b200.csrc import build
    d = tmp_path_factory.mktemp("fake_cuda")
    nvcc = build.nvcc()
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-O0", "-Xcicc", "-O0",
                    "-std=c++17", "-Xcompiler", "-fPIC", f"-I{REPO / 'include'}", "-c", "-o",
                    str(d / "api.o"), str(build.CSRC / "api.cu")], check=True)
    # -Bsymbolic: the runtime of this library, whatever else the process has loaded
    subprocess.run(["g++", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    f"-I{Path(nvcc).resolve().parent.parent / 'include'}", "-o",
                    str(d / "libtpo_host.so"), str(REPO / "tests" / "fake_cuda" / "runtime.cpp"),
                    str(d / "api.o")], check=True)
    return d / "libtpo_host.so"


@pytest.fixture
def host_lib(host_build, tmp_path):
    """A fresh copy each time: the library keeps what it learnt about a device."""
    from toptimization_b200 import _lib
    copy = tmp_path / f"{tmp_path.name}.so"
    copy.write_bytes(host_build.read_bytes())
    L = ctypes.CDLL(str(copy))
    for name, (res, args) in _lib._SIGS.items():
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    L.fake_log.restype = ctypes.c_char_p
    L.fake_limits.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_size_t]
    return L


def host_launches(L):
    """The launches since the last call, one dict each."""
    out = []
    for line in L.fake_log().decode().splitlines():
        dev, name, *kv = line.split()
        out.append({"dev": int(dev), "name": name,
                    **{k: int(v) for k, v in (x.split("=") for x in kv)}})
    return out
