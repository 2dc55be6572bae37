"""Column bases of a pair's images in FP32 (host build): formed in double-single
and rounded once they are the FP64 value to half a unit in the last place and
the 2^-45 of four double-single operations, also where the terms cancel; from
rounded inputs they are not, which is why the far images of unequal spheres use
the former."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "regularized-stokesian-dynamics_gb300", "csrc")


@pytest.fixture(scope="module")
def base(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("images") / "images_check.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                           os.path.join(ROOT, "tests", "cpp", "images_check.cpp"), "-o", so])
    f = ctypes.CDLL(so).images_check

    def run(R, A, nx, ny):
        R, A = np.ascontiguousarray(R, dtype=np.float64), np.asfortranarray(A, dtype=np.float64)
        out = np.zeros((2, 3), dtype=np.float32)
        f(R.ctypes.data_as(ctypes.c_void_p), A.ctypes.data_as(ctypes.c_void_p), nx, ny,
          out[0].ctypes.data_as(ctypes.c_void_p), out[1].ctypes.data_as(ctypes.c_void_p))
        return out.astype(np.float64)
    return run


@pytest.mark.parametrize("skew", [0.0, 0.37])
def test_column_bases(base, skew):
    rng = np.random.default_rng(3)
    worst_f = worst_s = 0.0
    for _ in range(400):
        L = rng.uniform(5.0, 30.0)
        A = L * np.array([[1.0, 0.0, skew], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]])
        R = rng.uniform(-0.5, 0.5, 3) * L
        nx, ny = (int(k) for k in rng.integers(-5, 6, 2))
        p = R + nx * A[:, 0] + ny * A[:, 1]
        size = np.abs(R) + np.abs(nx * A[:, 0]) + np.abs(ny * A[:, 1])
        pf, ps = base(R, A, nx, ny)
        ulp = np.spacing(np.abs(ps).astype(np.float32)).astype(np.float64)
        assert (np.abs(ps - p) <= 0.5 * ulp + 2.0 ** -45 * size).all()
        worst_f, worst_s = max(worst_f, (np.abs(pf - p) / ulp).max()), max(worst_s, (np.abs(ps - p) / ulp).max())
    assert worst_s <= 0.5 + 1e-3 < 1.0 < worst_f
