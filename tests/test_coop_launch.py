"""The PCG's cooperative launch where fewer CTAs can be resident than the device
has SMs (a process with part of the GPU): smaller grids are tried, other errors
come back as they are.  Host code against a fake runtime."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "regularized-stokesian-dynamics_gb300", "csrc")
TOO_LARGE, OUT_OF_MEMORY = 720, 2


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("coop") / "coop_check.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC,
                           "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "coop_check.cpp"), "-o", so])
    f = ctypes.CDLL(so).coop_check

    def run(grid, room, other=0):
        ran, left = ctypes.c_int(0), ctypes.c_int(0)
        return f(grid, room, other, ctypes.byref(ran), ctypes.byref(left)), ran.value, left.value
    return run


@pytest.mark.parametrize("grid,room,taken", [(152, 152, 152), (152, 151, 76), (152, 76, 76), (152, 20, 19), (152, 1, 1),
                                             (7, 2, 1), (1, 1, 1)])
def test_the_grid_is_halved_until_it_fits(check, grid, room, taken):
    assert check(grid, room) == (taken, 1, 0)


def test_errors_come_back(check):
    assert check(152, 0) == (-TOO_LARGE, 0, TOO_LARGE)
    assert check(152, 152, OUT_OF_MEMORY) == (-OUT_OF_MEMORY, 0, OUT_OF_MEMORY)


def test_the_pcg_launches_through_it():
    for name in os.listdir(CSRC):
        if name.endswith(".cu"):
            src = open(os.path.join(CSRC, name)).read()
            assert src.count("cudaLaunchCooperativeKernel") == src.count("rsd_coop_launch("), name
