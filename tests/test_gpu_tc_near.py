"""The one-launch chain between two diagonal blocks of the tensor-core Cholesky
(row panel tile, then the next diagonal tile), through rsd_potrf_f32_dev: next
blocks of 1, 4, 127 and 128 columns, inside a 512-wide panel and across its
end.  Tolerances of the tensor-core factor, ||U^T U - A|| / ||A||: 2e-3 (TF32)
and 2e-5 (3xTF32)."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.mark.parametrize("n", [129, 132, 255, 256, 257, 384, 512, 513, 641, 1028])
@pytest.mark.parametrize("prec,tol", [(1, 2e-3), (3, 2e-5)])
def test_factor(rsd, n, prec, tol):
    import torch
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, n))
    A = (x @ x.T / n + np.eye(n)).astype(np.float32)
    ld = (n + 3) // 4 * 4
    buf = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    buf[:, :n] = torch.tensor(A)
    assert rsd.potrf_f32_dev(rsd.Context(0), buf[:, :n].t(), prec=prec) == 0
    U = np.triu(buf[:, :n].t().cpu().numpy().astype(np.float64))
    assert np.linalg.norm(A - U.T @ U) <= tol * np.linalg.norm(A)
