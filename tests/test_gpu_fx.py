"""The fixed-point state-tile kernel behind CRS_MODE_FP64 (crs_fx.cu).

Tolerance: the FP64 modes' gross-rate scaled error of 1e-12.  Derived: an
exponent is a sum of at most twelve terms rounded to 2^-49, an exponential
adds 2^-49.5, so a rate is within 1.2e-14; the reference's own FP64
exponents (up to ~400, half an ulp 2.8e-14 per operation) carry the rest.
"""
import numpy as np
import pytest

from conftest import GOLDEN_CASES
from create_rate_subs_gb300 import synth
from oracle.oracle import Oracle, gross_scale, wdot_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TOL = 1e-12


def _wdot(mech, T, P, Y, mode="fp64"):
    from create_rate_subs_gb300.rates import RateSubs
    rs = RateSubs(mech)
    N = mech.n_species
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    w = rs.wdot(*d, mode=mode).cpu().numpy()
    return w, rs.status()


@pytest.mark.parametrize("case", GOLDEN_CASES)
def test_golden_states(case, golden):
    """Every rate form (PLOG, Chebyshev, REV, non-integer nu, negative A,
    several T_common, SRI, HIGH) on the edge states: T = T_common, extreme T
    and P, zero and one-hot Y, sum Y > 1."""
    mech, g = golden(case)
    w, status = _wdot(mech, g["T"], g["P"], g["Y"])
    G = gross_scale(mech.tables, g["fwd"], g["rev"], g["pm"])
    err = wdot_errors(w, g["wdot"], G)
    assert err["scaled"] <= TOL, err
    assert status == (0, 0)


# tiles of 32 states; 152 tiles fill the SMs once, 304 twice (the rule that
# picks 16 or 8 warps per CTA changes at 152)
@pytest.mark.parametrize("name,n", [("small", 1), ("small", 33), ("gri53", 31), ("gri53", 32),
                                    ("gri53", 152 * 32), ("gri53", 152 * 32 + 1),
                                    ("gri53", 305 * 32 + 5), ("features", 65),
                                    ("large561", 33)])
def test_tiles_and_states_outside_the_scheme(name, n, golden, synth_mech):
    """Partial tiles and both CTA sizes; every seventh state lies outside
    the fixed-point scheme (T beyond its intervals, a subnormal, negative or
    zero mass fraction) among regular ones."""
    mech = golden(name)[0] if name == "features" else synth_mech(name)
    N = mech.n_species
    T, P, Y = synth.make_states(N, n, seed=n + N)
    T[0::7] = 119.0
    T[1::21] = 6500.0
    Y[0, 2::7] = 5e-310
    Y[1, 3::7] = -1e-3
    Y[2, 4::7] = 0.0
    T[5::7] = 1000.0
    T[6::14] = 130.0
    ref = Oracle(mech.blob).eval(T, P, Y)
    G = gross_scale(mech.tables, ref["fwd"], ref["rev"], ref["pm"])
    fin = np.all(np.isfinite(ref["wdot"]) & np.isfinite(G), axis=0)
    w, status = _wdot(mech, T, P, Y)
    assert np.array_equal(np.all(np.isfinite(w), axis=0), fin)
    # at 119 K the reference's own exp(Kc) is subnormal (~1e-312): there the
    # general FP64 kernel, which forms 1/Kc as one exponential, is the judge
    cold = T < 120.0
    judge = np.where(cold, _wdot(mech, T, P, Y, "fp64_warp")[0], ref["wdot"])
    assert wdot_errors(w[:, fin], judge[:, fin], G[:, fin])["scaled"] <= TOL
    assert status == (0, int(np.sum(~np.isfinite(w))))


@pytest.mark.parametrize("name,n", [("gri53", 153 * 32), ("large561", 33)])
def test_scratch_under_capture_and_on_two_streams(name, n, synth_mech):
    """Launches whose net rates live in scratch: a handle's first call may be
    captured, a replay and calls on two streams at once give the eager bits."""
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech(name)
    N = mech.n_species
    sets = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
            for T, P, Y in (synth.make_states(N, n, seed=s) for s in (1, 2))]
    rs = RateSubs(mech)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = rs.wdot(*sets[0])
    eager = [rs.wdot(*d) for d in sets]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, eager[0])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for _ in range(8):
        for d, st in zip(sets, streams):
            with torch.cuda.stream(st):
                outs.append(rs.wdot(*d))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, eager[0])
    for k, o in enumerate(outs):
        assert torch.equal(o, eager[k % 2])
