"""Dynamic shared memory above 48 KB is a grant per kernel and device: a process
with contexts on two devices needs it on both, and threads with contexts of
their own must not share a flag.  The helper is run against a fake runtime
(no GPU), and no other place in the library asks for it."""
import ctypes
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "regularized-stokesian-dynamics_gb300", "csrc")


def test_granted_once_per_context_and_kernel(tmp_path):
    so = str(tmp_path / "smem_check.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC,
                           "-I", "/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "smem_check.cpp"), "-o", so])
    assert ctypes.CDLL(so).smem_check() == 0


def test_no_other_place_asks():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = open(path).read()
        assert "cudaFuncSetAttribute" not in src, path
        assert not re.search(r"^\s*static bool \w+\s*(=|\[)", src, re.M), path
