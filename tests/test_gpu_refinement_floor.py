"""Pairs so close that the residual of the mixed form's refinement stops at the
rounding of the velocities (gap 1e-8: R_lub cancels from ~1e8 times them): the
step is accepted there, by the stationary iteration or by flexible GMRES, with one
and with two right-hand sides, and matches the FP64 form to the mixed form's
1e-8.  Such steps returned RSD_ENOCONV."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


def close_pair(rsd, N, gap):
    """A packing whose closest pair is moved to the given gap."""
    pos, radii, L = rsd.configs.packing(N, 0.25, 0.02, seed=1, sweeps=20)
    d = pos[:, None] - pos[None]
    d -= np.round(d / L) * L
    r = np.sqrt((d ** 2).sum(-1))
    np.fill_diagonal(r, np.inf)
    i, j = np.unravel_index(r.argmin(), r.shape)
    e = d[i, j] / r[i, j] * (r[i, j] - 2.0 - gap) / 2.0
    pos[i] -= e
    pos[j] += e
    return pos, radii, L


@pytest.mark.parametrize("refinement", [0, 1])
@pytest.mark.parametrize("N,gap", [(32, 1e-6), (32, 1e-7), (32, 1e-8), (100, 1e-7)])
def test_floor_is_accepted(rsd, N, gap, refinement):
    pos, radii, L = close_pair(rsd, N, gap)
    tab, mu = rsd.LubTab(rsd.lubdat_dir()), rsd.mu_f_dimensionless(1.0)
    ctx = rsd.Context(0)
    ctx.set_refinement(refinement)
    for Fe in (None, np.random.default_rng(2).normal(size=6 * N)):
        step = lambda prec: rsd.STEPPER_Stokesian(ctx, tab, pos, radii, 0.0, 5e-4, [L] * 3, 1.0, mu, 1e-10, Fe=Fe,  # noqa: E731
                                                  precision=prec, max_iter=100)
        ref, g = step(rsd.PREC_FP64), step(rsd.PREC_MIXED)
        assert g["info"].info == 0 and g["info"].residual <= 1e-8
        for k in ("U_pos", "SijN"):
            assert np.abs(g[k] - ref[k]).max() <= 1e-8 * np.abs(ref[k]).max()
