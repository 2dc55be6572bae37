"""The FP32 Cholesky's diagonal-block kernel through rsd_potrf_f32_dev: sizes
at the edges of its thread tiles, its 32-row groups and the 128-wide block,
leading dimensions that rule out its vector accesses, and the index of the
first pivot that is not positive.  Tolerance: ||A - U^T U|| <= 16 n eps32 ||A||
(three times the n eps32 bound of an FP32 Cholesky, for reciprocals and square
roots of 2 ulp)."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float32).eps


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


def spd(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, n))
    return (x @ x.T / n + np.eye(n)).astype(np.float32)


@pytest.mark.parametrize("n,ld", [(1, 1), (2, 4), (31, 31), (32, 32), (33, 36), (127, 127), (128, 128), (128, 129),
                                  (129, 132), (200, 201)])
def test_factor(rsd, n, ld):
    import torch
    A = spd(n, n)
    buf = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    buf[:, :n] = torch.tensor(A)
    ctx = rsd.Context(0)
    assert rsd.potrf_f32_dev(ctx, buf[:, :n].t(), prec=0) == 0
    U = np.triu(buf[:, :n].t().cpu().numpy().astype(np.float64))
    assert np.linalg.norm(A - U.T @ U) <= 16 * n * EPS * np.linalg.norm(A)


@pytest.mark.parametrize("bad", [0, 1, 31, 32, 63, 126, 127, 128, 199])
@pytest.mark.parametrize("value", [-1.0, float("nan")])
def test_info(rsd, bad, value):
    import torch
    A = spd(200, 5)
    A[bad, bad] = value
    t = torch.tensor(A, device="cuda")
    assert rsd.potrf_f32_dev(rsd.Context(0), t.t(), prec=0) == bad + 1
