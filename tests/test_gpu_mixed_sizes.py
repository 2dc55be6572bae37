"""The mixed step against the plain FP64 one at the sizes where its padded
layout turns: one particle, sizes whose 6N or 11N is not a multiple of 4, both
sides of a 128-wide block of the stresslets (5N = 125, 130) and of the
512-wide blocks of the solves, one and two right-hand sides, equal and unequal
radii.  Tolerance: the mixed form's 1e-8."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.mark.parametrize("N,forces,unequal", [(1, False, False), (1, True, False), (2, False, False), (3, True, True),
                                              (13, False, False), (25, True, False), (26, False, False),
                                              (46, False, True), (47, True, False), (103, False, False)])
def test_mixed_matches_fp64(rsd, N, forces, unequal):
    T = 0.37
    pos, radii, L = rsd.configs.sheared_packing(N, 0.2, 0.01, 20268000 + N, T, sweeps=5)
    if unequal:
        radii = np.where(np.arange(N) % 2 == 0, 0.75, 1.0)
    Fe = np.random.default_rng(N).normal(size=6 * N) if forces else None
    ctx, tab = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir())
    mu = rsd.mu_f_dimensionless(1.0)
    a, b = (rsd.STEPPER_Stokesian(ctx, tab, pos, radii, T, 1e-3, [L, L, L], 1.0, mu, 1e-10, Fe=Fe, precision=p)
            for p in (rsd.PREC_MIXED, rsd.PREC_FP64))
    for k in ("U_pos", "SijN"):
        assert np.abs(a[k] - b[k]).max() <= 1e-8 * np.abs(b[k]).max(), k
    assert np.abs(a["conf"] - b["conf"]).max() <= 1e-10 * L
    assert np.abs(a["yeta_mu"] - b["yeta_mu"]).max() <= 1e-8 * np.abs(b["yeta_mu"]).max()
    assert a["info"].n_contact == b["info"].n_contact
