"""The PCG of the resistance solve at its edges: right-hand sides that hold a
NaN or an infinity are refused with RSD_ENAN (by the solve and by the FP64 step
that uses it), as the factorisation path refuses them; the solution may overwrite
the right-hand side."""
import ctypes

import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


@pytest.fixture(scope="module")
def system(rsd):
    import torch
    ctx, tab = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir())
    N = 27
    pos, radii, L = rsd.configs.packing(N, 0.30, 0.01, seed=20262110, sweeps=20)
    pos_t = torch.tensor(pos, dtype=torch.float64, device="cuda")
    radii_t = torch.tensor(radii, dtype=torch.float64, device="cuda")
    mu = rsd.mu_f_dimensionless(1.0)
    rpp, lat = rsd.resistance_pp_dev(ctx, tab, pos_t, radii_t, 0.0, [L, L, L], 1.0, mu, 1e-10)
    return dict(ctx=ctx, tab=tab, N=N, pos=pos, radii=radii, L=L, pos_t=pos_t, radii_t=radii_t, mu=mu, rpp=rpp, lat=lat,
                b=np.random.default_rng(3).normal(size=(2, 6 * N)))


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("mode", ["PC_NONE", "PC_FSAI"])
def test_nonfinite_right_hand_side(rsd, system, mode, value):
    import torch
    s = system
    for column in (0, 1):
        b = s["b"].copy()
        b[column, 7] = value
        with pytest.raises(rsd.RSDError) as e:
            rsd.pcg_dev(s["ctx"], None, getattr(rsd, mode), s["pos_t"], s["radii_t"], s["lat"], s["rpp"],
                        torch.tensor(b, device="cuda"))
        assert e.value.code == rsd.RSD_ENAN
    x, _, res = rsd.pcg_dev(s["ctx"], None, getattr(rsd, mode), s["pos_t"], s["radii_t"], s["lat"], s["rpp"],
                            torch.tensor(s["b"], device="cuda"))
    assert res <= 1e-12 and bool(torch.isfinite(x).all())


@pytest.mark.parametrize("mode", ["PC_NONE", "PC_FSAI"])  # PC_NONE: the factorisation
def test_step_with_a_nan_force(rsd, system, mode):
    s = system
    ctx = rsd.Context(0)
    ctx.set_rpp_solver(getattr(rsd, mode))
    Fe = np.zeros(6 * s["N"])
    Fe[4] = np.nan
    with pytest.raises(rsd.RSDError) as e:
        rsd.STEPPER_Stokesian(ctx, s["tab"], s["pos"], s["radii"], 0.0, 1e-3, [s["L"]] * 3, 1.0, s["mu"], 1e-10, Fe=Fe)
    assert e.value.code == rsd.RSD_ENAN


@pytest.mark.parametrize("mode", ["PC_NONE", "PC_JACOBI", "PC_FSAI"])
def test_solution_in_place_of_the_right_hand_side(rsd, system, mode):
    import torch
    s = system
    m = getattr(rsd, mode)
    b = torch.tensor(s["b"], device="cuda")
    ref, it0, _ = rsd.pcg_dev(s["ctx"], None, m, s["pos_t"], s["radii_t"], s["lat"], s["rpp"], b)
    it, res = ctypes.c_int32(0), ctypes.c_double(0.0)
    torch.cuda.synchronize()
    s["ctx"].check(rsd.library().rsd_lp_pcg_dev(s["ctx"].h, None, m, s["N"], s["pos_t"].data_ptr(),
                                                s["radii_t"].data_ptr(), ctypes.byref(s["lat"]), s["rpp"].data_ptr(),
                                                s["rpp"].stride(1), 2, b.data_ptr(), b.data_ptr(), 1e-12, 2000,
                                                ctypes.byref(it), ctypes.byref(res)))
    assert it.value == it0 and res.value <= 1e-12 and bool((b == ref).all())
    zero = torch.zeros_like(ref)  # no iteration: x is still written
    x, it, res = rsd.pcg_dev(s["ctx"], None, m, s["pos_t"], s["radii_t"], s["lat"], s["rpp"], zero)
    assert it == 0 and res == 0.0 and bool((x == 0).all())
