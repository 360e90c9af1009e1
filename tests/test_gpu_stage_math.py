"""The exponentials and divisions of the batched eval_rxn_rates and
get_rxn_pres_mod against CRS_MODE_FP64_STRICT, which evaluates the same
operations with CUDA's.

Tolerances: the exponents are the same numbers (a quotient by T is correctly
rounded either way), so a rate constant differs by its exponential's last
bits, 2 ulp (4.4e-16); a reverse rate by those of two; a fall-off factor by
those of about ten operations, times the slope of log10 F in log10 Pr (below
2): 1e-14.
"""
import numpy as np
import pytest

from create_rate_subs_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name,n", [("small", 1), ("gri53", 33), ("gri53", 4099),
                                    ("large561", 127)])
def test_stages_agree_with_the_strict_kernel(name, n, synth_mech):
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech(name)
    N = mech.n_species
    T, P, Y = synth.make_states(N, n, seed=n + N)
    T[1::9] = 1.0          # the end of the range of the division by T
    T[2::9] = 0.7          # below it
    T[3::9] = 1000.0
    T[4::9] = np.nextafter(2048.0, 0.0)  # a significand of ones
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    rs = RateSubs(mech)
    ref = rs.wdot_stages(*d, "fp64_strict")
    conc = rs.eval_conc(*d)[3]
    fwd, rev = rs.eval_rxn_rates(d[0], d[1], conc)
    pm = rs.get_rxn_pres_mod(d[0], d[1], conc)
    for got, want, tol in ((fwd, ref["fwd"], 5e-16), (rev, ref["rev"], 2e-15),
                           (pm, ref["pm"], 1e-14)):
        a, b = got.cpu().numpy(), want.cpu().numpy()
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        ok = np.isfinite(b) & (np.abs(b) > 1e-290)
        assert np.all(np.abs(a - b)[ok] <= tol * np.abs(b)[ok])
