"""The device-side waits of the FP64 products and of the PCG's grid barriers run
out without a fault when their bound is far below what the work needs: the
call returns RSD_ETIMEOUT, twice, and with the default bounds back the same
context gives the right answer."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


def timed_out(rsd, call):
    for _ in range(2):
        with pytest.raises(rsd.RSDError) as e:
            call()
        assert e.value.code == rsd.RSD_ETIMEOUT and "timed out" in str(e.value)


def test_fp64_products(rsd):
    n = 300
    G = np.random.default_rng(1).normal(size=(n, n))
    A = G @ G.T / n + np.eye(n)
    ctx = rsd.Context(0)
    ctx.set_wait_limits(tc_wait_ns=1)  # 1 ns: the first TMA load cannot land in time
    timed_out(rsd, lambda: rsd.MATREV(ctx, A))
    timed_out(rsd, lambda: rsd.CHOLESKY(ctx, A))
    ctx.set_wait_limits(0, 0)
    X, info = rsd.MATREV(ctx, A)
    ref = np.linalg.inv(A)
    assert info == 0 and np.abs(X - ref).max() <= 1e-13 * np.abs(ref).max()


def test_pcg_barriers(rsd):
    import torch
    N = 27
    pos, radii, L = rsd.configs.packing(N, 0.30, 0.01, seed=20262110, sweeps=20)
    pos_t, radii_t = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (pos, radii))
    ctx = rsd.Context(0)
    rpp, lat = rsd.resistance_pp_dev(ctx, rsd.LubTab(rsd.lubdat_dir()), pos_t, radii_t, 0.0, [L, L, L], 1.0,
                                     rsd.mu_f_dimensionless(1.0), 1e-10)
    b = torch.tensor(np.random.default_rng(3).normal(size=6 * N), device="cuda")
    solve = lambda: rsd.pcg_dev(ctx, None, rsd.PC_FSAI, pos_t, radii_t, lat, rpp, b)  # noqa: E731
    ref = solve()[0]
    ctx.set_wait_limits(tri_spin_polls=1)  # one poll: the CTAs do not arrive within it
    timed_out(rsd, solve)
    ctx.set_wait_limits(0, 0)
    x, it, res = solve()
    assert it > 0 and res <= 1e-12 and bool((x == ref).all())
