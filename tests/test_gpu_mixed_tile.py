"""The state tiles behind CRS_MODE_MIXED (crs_mixed_tile.cu) against the
kernels that evaluate every reaction by the general code.

Tolerance: the exponents agree to about 1e-12, which may move the FP32
roundings of a rate by one unit (2^-24 in the reduced exponent, in the
exponential and in the product: 1.8e-7) and of its fall-off factor likewise;
relative to the gross rates 4e-7 covers both.
"""
import numpy as np
import pytest

from conftest import GOLDEN_CASES
from create_rate_subs_gb300 import synth
from oracle.oracle import Oracle, gross_scale, wdot_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TOL = 4e-7


# one tile; partial tiles; clusters of 8, 4 and 2 CTAs per tile; one CTA per
# tile; whole waves and a remainder (152 SMs, three CTAs each)
@pytest.mark.parametrize("name,n", [("small", 1), ("small", 4099), ("gri53", 31), ("gri53", 33),
                                    ("gri53", 38 * 32), ("gri53", 70 * 32 + 1),
                                    ("gri53", 152 * 32), ("gri53", 456 * 32 + 7),
                                    ("large561", 33), ("large561", 153 * 32 + 5)]
                         + [(c, 67) for c in GOLDEN_CASES])
def test_agrees_with_the_general_kernels(name, n, golden, synth_mech):
    """States with zero, negative and subnormal mass fractions, temperatures
    at and beyond the polynomials' ends and zero pressure among regular ones."""
    from create_rate_subs_gb300.rates import RateSubs
    mech = golden(name)[0] if name in GOLDEN_CASES else synth_mech(name)
    N = mech.n_species
    T, P, Y = synth.make_states(N, n, seed=n + N)
    T[0::7] = 119.0
    T[1::21] = 6500.0
    T[5::7] = 1000.0
    P[2::33] = 0.0
    Y[0, 2::7] = 5e-310
    Y[1, 3::7] = -1e-3
    Y[2, 4::7] = 0.0
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    rs = RateSubs(mech)
    w = rs.wdot(*d, mode="mixed").cpu().numpy()
    status = rs.status()
    ref = rs.wdot(*d, mode="mixed_warp").cpu().numpy()
    o = Oracle(mech.blob).eval(T, P, Y)
    G = gross_scale(mech.tables, o["fwd"], o["rev"], o["pm"])
    assert np.array_equal(np.isfinite(w), np.isfinite(ref))
    assert status == (0, int(np.sum(~np.isfinite(w))))
    fin = np.all(np.isfinite(w) & np.isfinite(G), axis=0)
    assert wdot_errors(w[:, fin], ref[:, fin], G[:, fin])["scaled"] <= TOL
