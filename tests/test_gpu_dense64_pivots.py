"""A pivot that is not positive at every place of a diagonal block of the FP64
Cholesky: the index comes back as LAPACK's each time (the CTA's warps leave the
block together), and the context factors the next matrix as before."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 100])
def test_every_pivot(n):
    ge._load_build_module().build()
    rsd = ge.load_package()
    ctx = rsd.Context(0)
    rng = np.random.default_rng(n)
    G = rng.normal(size=(n, n))
    A = G @ G.T / n + np.eye(n)
    ref = np.linalg.inv(A)
    for bad in range(n):
        B = A.copy()
        B[bad, bad] = -1.0
        assert rsd.MATREV(ctx, B)[1] == bad + 1
    X, info = rsd.MATREV(ctx, A)
    assert info == 0 and np.abs(X - ref).max() <= 1e-13 * np.abs(ref).max()
