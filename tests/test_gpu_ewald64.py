"""The FP64 grand mobility's pair kernel against the oracle at the sizes where
its dispatch turns: one pair, fewer pairs than a block takes, both sides of
the 8192 pairs that separate 32 lanes per pair from 8 (N = 128, 129), equal
and unequal radii, cells of several skews, and an EWS_ERR loose enough that
the reference's cubes cut the sum (1e-4: the whole cubes are summed) beside
the usual one (spheres at another splitting parameter).  Tolerance: 1e-12 of
the largest entry, the bar of every mobility test."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as o

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.mark.parametrize("N,phi,T,ews,unequal", [
    (1, 0.05, 0.37, 1e-10, False), (2, 0.05, 0.0, 1e-10, False), (3, 0.10, 0.81, 1e-10, True),
    (9, 0.20, 0.5, 1e-4, False), (9, 0.20, 0.25, 1e-4, True), (27, 0.30, 0.97, 1e-10, True),
    (128, 0.25, 0.6, 1e-10, False), (129, 0.25, 0.6, 1e-10, False), (129, 0.20, 0.13, 1e-10, True),
    (129, 0.20, 0.13, 1e-4, False)])
def test_mobility_matches_oracle(rsd, N, phi, T, ews, unequal):
    pos, radii, L = rsd.configs.sheared_packing(N, phi, 0.01, 20267000 + N, T, sweeps=5)
    if unequal:
        radii = np.where(np.arange(N) % 3 == 0, 0.7, np.where(np.arange(N) % 3 == 1, 1.0, 0.85))
    ctx, mu = rsd.Context(0), rsd.mu_f_dimensionless(1.0)
    lat = rsd.SET_LATTICE_SKEW(T, [L, L, L], 1.0)
    got = rsd.PER_GRPERY_INV_FRI(ctx, pos, radii, lat, ews, mu)
    ref = o.split_mobility(o.per_grpery_inv_fri(pos, radii, o.set_lattice_skew(T, [L, L, L], 1.0), ews, mu)[0], N)
    for g, r in zip(got, ref):
        assert np.abs(g - r).max() <= 1e-12 * np.abs(ref[0]).max()
