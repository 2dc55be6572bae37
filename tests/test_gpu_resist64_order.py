"""A grand mobility within rounding of a singular one, whose FP64 Cholesky
factor exists in the reference's order (forces before stresslets) and not with
the stresslets first, as the resistance solve orders it: the solve then takes
the reference's order.  One particle, M the identity but for a force-stresslet
pair [a b; b c] whose pivots are a, c - l b > 0 with l = b rn(1 / a) in the one
order and c, a - p^2 <= 0 with p = b rn(1 / rn(sqrt c)) in the other.  With e the
pair's strain and no lubrication the velocity of the coupled component tends to
-e / l (R00 = 1 / a + l^2 / d, R06 = -l / d, d ~ 1e-16); the others are F."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu

TRIPLES = [("0x1.0a7d3da94ecdep+0", "0x1.08764f6c2685ep-1", "0x1.067353b08f20ep-2"),
           ("0x1.d0dbc74d47003p+0", "0x1.0166f0d1577d2p-1", "0x1.1d0ee1322d86cp-3"),
           ("0x1.af7fadf361287p+0", "0x1.26847fc6f339cp+0", "0x1.920b19354cfc0p-1")]


@pytest.mark.parametrize("triple", TRIPLES)
def test_reference_order_is_taken(triple):
    ge._load_build_module().build()
    rsd = ge.load_package()
    a, b, c = (float.fromhex(x) for x in triple)
    p = b * (1.0 / np.sqrt(c))
    assert a - p * p <= 0.0
    APP, APQ, AQQ = np.eye(6), np.zeros((6, 5)), np.eye(5)
    APP[0, 0], APQ[0, 0], AQQ[0, 0] = a, b, c
    Fe, EIN = np.arange(1.0, 7.0), np.array([0.75, -1.0, 0.5, 2.0, 1.0])
    ctx = rsd.Context(0)
    zero = np.zeros
    for _ in range(2):  # the second call starts from the first one's buffers
        out = rsd.STEPPER_NOGmres(ctx, APP, APQ, AQQ, zero((6, 6)), zero((6, 5)), zero((5, 5)), Fe, EIN, zero(6), zero(3))
        assert out["info"] == 0
        l = b * (1.0 / a)
        assert abs(out["U_par"][0] + EIN[0] / l) <= 1e-12 * abs(EIN[0] / l)
        assert np.abs(out["U_par"][1:] - Fe[1:]).max() <= 1e-14 * 6
        assert np.isfinite(out["SijN_hyd"]).all() and np.abs(out["SijN_hyd"][1:] + EIN[1:]).max() <= 1e-14 * 2
    # a pair that fails in both orders: the index of the reference's order
    AQQ[0, 0] = 0.5 * c
    assert rsd.STEPPER_NOGmres(ctx, APP, APQ, AQQ, zero((6, 6)), zero((6, 5)), zero((5, 5)), Fe, EIN, zero(6),
                               zero(3))["info"] == 7
