"""rsd_ctx_set_mixed_real_passes at a size whose image sums are dealt out over
slices by default: 2 to 4 passes take the kernel they name (one launch fewer
than the slices), and the step is the same to the rounding of the sums (FP32
terms in another order: 1e-9 of the largest stresslet, a tenth of the mixed
form's bound)."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [20, 64])
def test_passes_are_taken(N):
    ge._load_build_module().build()
    rsd = ge.load_package()
    ctx, tab, lib = rsd.Context(0), rsd.LubTab(rsd.lubdat_dir()), rsd.library()
    pos, radii, L = rsd.configs.packing(N, 0.25, 0.01, seed=20262120, sweeps=10)
    out, launches = {}, {}
    for passes in (1, 2, 3, 4):
        ctx.set_mixed_real_passes(passes)
        for _ in range(2):  # the first step also launches what is built once
            n0 = lib.rsd_launch_count()
            out[passes] = rsd.STEPPER_Stokesian(ctx, tab, pos, radii, 0.0, 1e-3, [L] * 3, 1.0,
                                                rsd.mu_f_dimensionless(1.0), 1e-10, precision=rsd.PREC_MIXED)
            launches[passes] = lib.rsd_launch_count() - n0
    its = {p: o["info"].iterations for p, o in out.items()}
    for p in (2, 3, 4):
        if its[p] == its[1]:
            assert launches[p] == launches[1] - 1
        for k in ("U_pos", "SijN"):
            assert np.abs(out[p][k] - out[1][k]).max() <= 1e-9 * np.abs(out[1][k]).max()
    assert any(its[p] == its[1] for p in (2, 3, 4))
