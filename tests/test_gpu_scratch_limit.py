"""The FP64 inverse and resistance where the memory for their workspaces cannot
be had: they work in place of the matrix, and fail only without room for that."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


def stiff(n, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    A = (q * np.exp(rng.uniform(0.0, 2.0, n))) @ q.T
    for i in range(0, n - 9, 6):
        v, e = np.zeros(n), rng.normal(size=3)
        v[i:i + 3] = e / np.linalg.norm(e)
        v[i + 6:i + 9] = -v[i:i + 3]
        A += 1e7 * np.outer(v, v)
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("n", [65, 512, 513, 1100, 1536])  # one block of 512 columns, two, three
def test_inverse_in_place(rsd, n):
    """||A X - I|| <= n eps ||A|| ||X||, the bound of the inverse in its own memory,
    and once more for the product taken here."""
    A = stiff(n, n)
    ctx = rsd.Context(0)
    W = (n + 63) // 64 * 64
    # the matrix, the diagonal inverses, and a tenth more than the workspaces in place take
    ctx.set_scratch_limit(8 * n * n + 8 * 64 * W + int(1.1 * 36 * 512 * n) + 14 * 512 * 512)
    X, info = rsd.MATREV(ctx, A)
    E = A @ X - np.eye(n)
    assert info == 0 and np.linalg.norm(E) <= 2 * n * EPS * np.linalg.norm(A) * np.linalg.norm(X)
    assert np.array_equal(X, X.T)
    fresh = rsd.Context(0)
    fresh.set_scratch_limit(8 * n * n // 2)
    with pytest.raises(rsd.RSDError) as e:
        rsd.MATREV(fresh, A)
    assert e.value.code == rsd.RSD_ENOMEM
    fresh.set_scratch_limit(0)
    X2, info = rsd.MATREV(fresh, A)
    assert info == 0 and np.abs(X2 - X).max() <= 4 * n * EPS * np.linalg.norm(A) * np.linalg.norm(X) ** 2


@pytest.mark.parametrize("rpp", [False, True])
def test_step_in_less_memory(rsd, rpp):
    """N = 160: limits from the grand mobility (25 MB) to more than all workspaces.
    In between, over 25 MB, only M^-1 in place of M fits, then over 6 MB the
    factor of M' but not V beside the inverse.  The resistance matrices' condition
    numbers are below 1e4, so two backward stable forms agree to 1e4 n eps."""
    N = 160
    pos, radii, L = rsd.configs.packing(N, 0.3, 1e-2, 7)
    mu = rsd.mu_f_dimensionless(1.0)
    tab = rsd.LubTab(rsd.lubdat_dir())

    def step(limit):
        ctx = rsd.Context(0)
        ctx.set_scratch_limit(limit)
        if rpp:
            ctx.set_rpp_solver(rsd.PC_BLOCK_JACOBI)
        o = rsd.STEPPER_Stokesian(ctx, tab, pos.copy(), radii, 0.0, 5e-4, [L, L, L], 1.0, mu, 1e-10)
        assert o["rc"] == 0 and o["info"].info == 0
        return o["U_pos"], o["SijN"]

    U, S = step(0)
    n, P = 11 * N, 6 * N
    bound = 1e4 * n * EPS
    taken = 0
    for limit in np.linspace(8 * n * n, 8 * (3 * n * n + 12 * P * P), 24).astype(np.int64):
        try:
            u, s = step(int(limit))
        except rsd.RSDError as e:
            assert e.code == rsd.RSD_ENOMEM
            continue
        assert np.abs(u - U).max() <= bound * np.abs(U).max()
        assert np.abs(s - S).max() <= bound * np.abs(S).max()
        taken += 1
    assert taken >= 10
