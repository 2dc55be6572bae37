"""The sliced pair sums of a small system's mixed mobility (equal radii)
against the plain FP64 step: one pair, sizes around the 32 x 4 pair tiles and
the 16 pairs of a joining block, and both sides of the size (~190) above which
the sums are not sliced.  Tolerance: the mixed form's 1e-8."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.mark.parametrize("N,T", [(2, 0.0), (6, 0.5), (17, 0.0), (32, 0.31), (33, 0.5), (64, 0.0), (65, 0.2),
                                 (129, 0.43), (180, 0.1), (200, 0.1)])
def test_step_matches_fp64(rsd, N, T):
    pos, radii, L = rsd.configs.sheared_packing(N, 0.25, 0.01, 20269000 + N, T, sweeps=5)
    ctx, tab = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir())
    mu = rsd.mu_f_dimensionless(1.0)
    a, b = (rsd.STEPPER_Stokesian(ctx, tab, pos, radii, T, 1e-3, [L, L, L], 1.0, mu, 1e-10, precision=p)
            for p in (rsd.PREC_MIXED, rsd.PREC_FP64))
    for k in ("U_pos", "SijN", "yeta_mu"):
        assert np.abs(a[k] - b[k]).max() <= 1e-8 * np.abs(b[k]).max(), k
