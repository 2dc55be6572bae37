"""Branches of the step that few systems reach: overlap corrections on a system
whose image sums are dealt out over slices, unequal radii under other splits,
truncations and splitting parameters than the defaults, and two contexts stepping
at once in the FP64 form.  Mixed against FP64 to the mixed form's 1e-8; the FP64
form against itself, alone, exactly."""
import threading

import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rsd():
    ge._load_build_module().build()
    return ge.load_package()


def step(rsd, ctx, tab, pos, radii, L, precision):
    return rsd.STEPPER_Stokesian(ctx, tab, pos, radii, 0.0, 1e-3, [L] * 3, 1.0, rsd.mu_f_dimensionless(1.0), 1e-10,
                                 precision=precision)


def close(a, b, tol):
    for k in ("U_pos", "SijN"):
        assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), k


@pytest.mark.parametrize("method", [1, 2])
def test_overlap_correction_on_a_sliced_system(rsd, method):
    """One overlapping pair (r = 1.98).  With Yamakawa's blocks its mobility is
    not positive definite (smallest eigenvalue -0.028 by the oracle): both forms
    report it.  The regularized blocks change the stresslets by a quarter."""
    pos, radii, L = rsd.configs.packing(24, 0.20, 0.02, seed=20262140, sweeps=10)
    d = pos[:, None] - pos[None]
    d -= np.round(d / L) * L
    r = np.sqrt((d ** 2).sum(-1))
    np.fill_diagonal(r, np.inf)
    i, j = np.unravel_index(r.argmin(), r.shape)
    pos[i] -= d[i, j] / r[i, j] * (r[i, j] - 1.98)
    ctx, tab = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir())
    plain = step(rsd, ctx, tab, pos, radii, L, rsd.PREC_FP64)
    ctx.set_correction_method(method)
    ref, mixed = (step(rsd, ctx, tab, pos, radii, L, p) for p in (rsd.PREC_FP64, rsd.PREC_MIXED))
    if method == 1:
        assert ref["info"].info > 0 and mixed["info"].info > 0
        ctx.set_correction_method(0)  # and the context steps on
        close(step(rsd, ctx, tab, pos, radii, L, rsd.PREC_MIXED), plain, 1e-8)
        return
    assert ref["info"].n_contact == mixed["info"].n_contact == 1
    assert np.abs(ref["SijN"] - plain["SijN"]).max() > 0.1 * np.abs(ref["SijN"]).max()
    close(mixed, ref, 1e-8)


@pytest.mark.parametrize("setting", [("set_mixed_split", (6.0, 2)), ("set_mixed_split", (5.0, 1)),
                                     ("set_mixed_truncation", (6.5, 36.0)), ("set_mixed_lambda_scale", (1.0,)),
                                     ("set_mixed_lambda_scale", (1.5,)), ("set_mixed_lambda_scale", (2.1,))])
@pytest.mark.parametrize("N", [33, 70])
def test_unequal_radii_under_other_settings(rsd, N, setting):
    pos, radii, L = rsd.configs.packing(N, 0.25, 0.02, seed=20262141, sweeps=10)
    radii = np.where(np.arange(N) % 3 == 0, 0.8, radii)  # smaller: no overlaps
    ctx, tab = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir())
    getattr(ctx, setting[0])(*setting[1])
    close(step(rsd, ctx, tab, pos, radii, L, rsd.PREC_MIXED), step(rsd, ctx, tab, pos, radii, L, rsd.PREC_FP64), 1e-8)


def test_two_contexts_at_once_in_fp64(rsd):
    jobs = []
    for N in (40, 90):
        pos, radii, L = rsd.configs.packing(N, 0.25, 0.02, seed=20262142 + N, sweeps=10)
        jobs.append((rsd.Context(0), rsd.LubTab(rsd.lubdat_dir()), pos, radii, L))
    ref = [step(rsd, *j, rsd.PREC_FP64) for j in jobs]
    out, errors = [[], []], []

    def work(k):
        try:
            for _ in range(10):
                out[k].append(step(rsd, *jobs[k], rsd.PREC_FP64))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k in range(2):
        assert len(out[k]) == 10
        for o in out[k]:
            for key in ("U_pos", "SijN", "conf"):
                assert np.array_equal(o[key], ref[k][key])
