"""Positions many cells outside the primary one (a driver that keeps unwrapped
coordinates): every entry point takes minimum images, so whole multiples of the
lattice vectors change the results by the rounding of the positions only: 1e6
cells of ~10 leave 1e-9 of a radius, which gaps of 0.02 turn into 1e-7 of the
lubrication blocks; the others move by less."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    ge._load_build_module().build()
    rsd = ge.load_package()
    N = 60
    pos, radii, L = rsd.configs.packing(N, 0.35, 0.02, seed=20262130, sweeps=30)
    k = np.random.default_rng(5).integers(-10 ** 6, 10 ** 6, size=(N, 3))
    return rsd, rsd.Context(0), rsd.LubTab(rsd.lubdat_dir()), pos, pos + k * L, radii, L, rsd.mu_f_dimensionless(1.0)


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def test_lubrication(case):
    rsd, ctx, tab, pos, far, radii, L, mu = case
    lat = rsd.SET_LATTICE_SKEW(0.0, [L] * 3, 1.0)
    a = rsd.lubmxcalc(ctx, tab, pos, radii, lat, mu)
    b = rsd.lubmxcalc(ctx, tab, far, radii, lat, mu)
    assert a[3] == b[3]
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x != 0.0, y != 0.0) and rel(y, x) <= 1e-6


def test_fp64_mobility(case):
    rsd, ctx, tab, pos, far, radii, L, mu = case
    lat = rsd.SET_LATTICE_SKEW(0.0, [L] * 3, 1.0)
    a = rsd.PER_GRPERY_INV_FRI(ctx, pos, radii, lat, 1e-10, mu)
    b = rsd.PER_GRPERY_INV_FRI(ctx, far, radii, lat, 1e-10, mu)
    for x, y in zip(a, b):
        assert rel(y, x) <= 1e-7


def test_preconditioner_graph(case):
    import torch
    rsd, ctx, tab, pos, far, radii, L, mu = case
    t = lambda x: torch.tensor(x, dtype=torch.float64, device="cuda")  # noqa: E731
    rpp, lat = rsd.resistance_pp_dev(ctx, tab, t(pos), t(radii), 0.0, [L] * 3, 1.0, mu, 1e-10)
    b = t(np.random.default_rng(6).normal(size=6 * len(radii)))
    x, it, _ = rsd.pcg_dev(ctx, None, rsd.PC_FSAI, t(pos), t(radii), lat, rpp, b)
    y, it2, res = rsd.pcg_dev(ctx, None, rsd.PC_FSAI, t(far), t(radii), lat, rpp, b)
    assert it2 == it and res <= 1e-12 and bool((x == y).all())
