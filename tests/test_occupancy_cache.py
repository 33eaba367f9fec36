"""The occupancy cache (cpabdiffeo_b200/csrc/cpab_occupancy.h): a program that
launches at many sizes asks for each once, and its memory is bounded.  CPU only."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("occupancy") / "liboccupancyhost.so"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "cpabdiffeo_b200" / "csrc"),
                    str(ROOT / "tests" / "occupancy_host.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.occupancy_queries.restype = C.c_long
    return lib


@pytest.mark.parametrize("kernels,sizes", [(1, 1), (1, 65), (4, 32), (20, 150)])
def test_each_size_is_asked_for_once(lib, kernels, sizes):
    assert lib.occupancy_queries(kernels, sizes, 5) == kernels * sizes


def test_bounded(lib):
    assert lib.occupancy_queries(1, 4096, 2) == 4096
    assert lib.occupancy_queries(1, 10000, 1) == 10000  # (starts anew twice; answers stay right)
