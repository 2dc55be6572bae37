"""The FP32 Cholesky at the ends of FP32's range, through rsd_potrf_f32_dev: the
factor of a matrix times a power of four is the matrix's factor times that of
two, to the factorisation's own bound, 16 n eps32 ||A||, with pivots above 2^126
and below 2^-110; sizes of one ragged block, one whole block, and several."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float32).eps


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.mark.parametrize("power", [126, -112])
@pytest.mark.parametrize("n", [20, 127, 128, 200])
def test_factor(rsd, n, power):
    import torch
    x = np.random.default_rng(n).normal(size=(n, n))
    A = (x @ x.T / n + np.eye(n))
    A = (A * (1.9 / np.diag(A).max())).astype(np.float32)
    t = torch.tensor(A * np.float32(2.0) ** power, device="cuda")
    assert bool(torch.isfinite(t).all())
    assert rsd.potrf_f32_dev(rsd.Context(0), t.t(), prec=0) == 0
    U = np.triu(t.t().cpu().numpy().astype(np.float64)) * 2.0 ** (-power // 2)
    assert np.linalg.norm(A - U.T @ U) <= 16 * n * EPS * np.linalg.norm(A)
