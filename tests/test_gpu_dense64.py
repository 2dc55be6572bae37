"""The FP64 factorisations on tensor cores (digit-sliced products) against
LAPACK in FP64 at the sizes where they can go wrong: one panel, its edges
(64), the edges of a 128-column tile, ragged last panels and ragged last pairs
of the recursive inverse, several drains of the accumulators, and columns of
very different scales.  Tolerances: the inverse of a matrix of condition
number c differs from LAPACK's by at most about n c eps of its norm in either
computation; 10 n c eps (and 1e-14) bound the difference.  The factor is held
by ||A - L L^T|| <= 10 n eps ||A||."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


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


@pytest.mark.parametrize("n,cond", [(1, 1.0), (5, 10.0), (63, 1e2), (64, 1e2), (65, 1e4), (127, 20.0), (128, 20.0),
                                    (129, 1e5), (192, 1e3), (193, 1e3), (320, 20.0), (704, 1e4), (1375, 20.0)])
def test_factor_and_inverse(rsd, ctx, n, cond):
    A = spd(n, cond, 100 + n)
    L = rsd.CHOLESKY(ctx, A)
    assert np.abs(np.triu(L, 1)).max(initial=0.0) == 0.0
    assert np.linalg.norm(A - L @ L.T) <= 10 * n * EPS * np.linalg.norm(A)
    inv, info = rsd.MATREV(ctx, A)
    assert info == 0
    ref = np.linalg.inv(A)
    assert np.abs(inv - inv.T).max() == 0.0
    assert np.linalg.norm(inv - ref) <= max(10 * n * cond * EPS, 1e-14) * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [70, 260])
def test_scaled_columns(rsd, ctx, n):
    """D A D with D over 12 orders: the factor scales with D."""
    A = spd(n, 10.0, 7 + n)
    D = 10.0 ** np.random.default_rng(n).uniform(-6, 6, n)
    L = rsd.CHOLESKY(ctx, A * D[:, None] * D[None, :])
    ref = np.linalg.cholesky(A)
    assert np.abs(L / D[:, None] - ref).max() <= 100 * n * EPS


@pytest.mark.parametrize("n,bad", [(10, 4), (100, 0), (100, 63), (100, 64), (200, 199)])
def test_info_and_nonfinite(rsd, ctx, n, bad):
    A = spd(n, 10.0, n)
    A[bad, bad] = -1.0
    assert rsd.MATREV(ctx, A)[1] == bad + 1
    A[bad, bad] = np.nan
    assert rsd.MATREV(ctx, A)[1] == bad + 1
    if bad > 64:  # a NaN off the first panel's diagonal reaches the pivot it feeds
        A = spd(n, 10.0, n)
        A[3, bad] = A[bad, 3] = np.nan
        assert rsd.MATREV(ctx, A)[1] == bad + 1


@pytest.mark.parametrize("N", [1, 7, 13])
def test_resistance_chain(rsd, ctx, N):
    """arrangement and STEPPER_NOGmres on a random SPD mobility."""
    p, q = 6 * N, 5 * N
    G = spd(11 * N, 20.0, 40 + N)
    Z = spd(11 * N, 1e3, 50 + N) * 5.0
    rng = np.random.default_rng(N)
    Fe, EIN, Fi, conf, ub = (rng.normal(size=k) for k in (p, q, p, 3 * N, 3 * N))
    out = rsd.STEPPER_NOGmres(ctx, G[:p, :p], G[:p, p:], G[p:, p:], Z[:p, :p], Z[:p, p:], Z[p:, p:], Fe, EIN, Fi, conf,
                              ub)
    R = np.linalg.inv(G) + Z
    RPP, RPQ, RQQ = R[:p, :p], R[:p, p:], R[p:, p:]
    UB = np.concatenate([ub, np.zeros(3 * N)])
    rel = lambda a, b: np.abs(a - b).max() / np.abs(b).max()  # noqa: E731
    assert rel(out["U_par"], np.linalg.solve(RPP, Fe + RPQ @ EIN)) <= 1e-11
    assert rel(out["SijN_hyd"], RPQ.T @ np.linalg.solve(RPP, RPQ @ EIN) - RQQ @ EIN) <= 1e-11
    assert rel(out["SijN_B"], RPQ.T @ UB) <= 1e-11
    assert rel(out["RPP"], np.linalg.inv(RPP)) <= 1e-11
    mu, info = rsd.arrangement(ctx, RPP, RPQ, RQQ)
    assert info == 0 and rel(mu, RPQ.T @ np.linalg.solve(RPP, RPQ) - RQQ) <= 1e-11
