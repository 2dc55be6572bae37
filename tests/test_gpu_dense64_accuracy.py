"""Accuracy of the FP64 factorisations on ill-conditioned matrices, against
what substitution with multiply-adds in FP64 keeps whatever the condition
number: residuals of some n eps of the operands' norms."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.fixture(scope="module")
def ctx(rsd):
    return rsd.Context(0)


def spd(n, cond, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    a = (q * np.exp(rng.uniform(-np.log(cond), 0.0, n))) @ q.T
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("N", [1, 11, 43])  # 6 N = 6, 66, 258: one block, ragged second block, ragged second panel
def test_many_right_hand_sides(rsd, ctx, N):
    """arrangement with RPQ = A X0, condition 1e10: RPQ^T A^-1 RPQ = X0^T A X0.
    With (A + D) X = RPQ exactly, |D| <= n eps |A|, the result moves by X0^T D X0
    and the roundings of RPQ and of the product, n eps |X0|^T |A| |X0| each."""
    p, q = 6 * N, 5 * N
    A = spd(p, 1e10, N)
    X0 = np.random.default_rng(N).normal(size=(p, q))
    B = A @ X0
    mu, info = rsd.arrangement(ctx, A, B, np.zeros((q, q)))
    ref = (B.T.astype(np.longdouble) @ X0).astype(np.float64)
    size = np.abs(X0).T @ np.abs(A) @ np.abs(X0)
    assert info == 0 and np.abs(mu - ref).max() <= 3 * p * EPS * size.max()


def stiff_pairs(n, gap, seed):
    """A well-conditioned matrix with a spring 1 / gap along a random axis between
    neighbouring bodies of six unknowns, as lubrication adds one."""
    rng = np.random.default_rng(seed)
    A = spd(n, 10.0, seed)
    for i in range(0, n - 9, 6):
        v, e = np.zeros(n), rng.normal(size=3)
        v[i:i + 3] = e / np.linalg.norm(e)
        v[i + 6:i + 9] = -v[i:i + 3]
        A += np.outer(v, v) / gap
    return A


@pytest.mark.parametrize("n", [65, 128, 300, 577])  # ragged and whole last blocks, one to three outer panels
def test_factor_residual(rsd, ctx, n):
    """|A - L L^T| <= n eps sqrt(A_ii A_jj), Cholesky's bound, on stiff pairs."""
    A = stiff_pairs(n, 1e-8, n)
    L = rsd.CHOLESKY(ctx, A).astype(np.longdouble)
    d = np.sqrt(np.diag(A))
    assert np.abs((A - L @ L.T) / np.outer(d, d)).max() <= n * EPS


@pytest.mark.parametrize("make,n,x", [(stiff_pairs, 129, 1e-8), (stiff_pairs, 300, 1e-8), (stiff_pairs, 391, 1e-7),
                                      (spd, 300, 1e12), (spd, 520, 1e12)])
def test_inverse_residual(rsd, ctx, make, n, x):
    """||A X - I|| <= n eps ||A|| ||X||: columns of the inverse by substitution."""
    A = make(n, x, n)
    X, info = rsd.MATREV(ctx, A)
    E = (A.astype(np.longdouble) @ X - np.eye(n)).astype(np.float64)
    assert info == 0 and np.linalg.norm(E) <= n * EPS * np.linalg.norm(A) * np.linalg.norm(X)


def test_digits_of_one_sign(rsd, ctx):
    """Columns whose lower digits are all -128, so that the digit products of
    every weight add up with one sign over all 256 terms, while the products
    themselves cancel: A = [I B; B^T C], B exact in 56 bits, whose factor holds
    C - B^T B in its last block.  Off the diagonal B^T B is near -1; the weights
    left out may come to 256 2^-61, its rounding and those of the last block's
    factor to 4 eps."""
    tail = sum(2.0 ** (-8 * i) for i in range(1, 7))
    B = np.full((256, 2), 0.5 - tail)
    B[::2, 1] = -(0.5 + tail)
    B[255] = 0.75
    A = np.eye(258)
    A[:256, 256:], A[256:, :256] = B, B.T
    A[256:, 256:] = B.T @ B + np.eye(2)
    L = rsd.CHOLESKY(ctx, A)
    assert np.array_equal(L[256:, :256], B.T)
    R = A[256:, 256:].astype(np.longdouble) - L[256:].astype(np.longdouble) @ L[256:].T.astype(np.longdouble)
    assert abs(float(R[0, 1])) <= 256 * 2.0 ** -61 + 4 * EPS
