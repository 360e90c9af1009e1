"""States that the fixed-point state tiles (crs_fx.cu) leave to the general FP64
arithmetic: any number of them in a tile, alone or among others, and rates
whose factors are far below the normal range.

Tolerance: the FP64 modes' gross-rate scaled error of 1e-12.
"""
import numpy as np
import pytest

from create_rate_subs_gb300 import synth
from oracle.oracle import Oracle, gross_scale, wdot_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# launches by clusters, one tile per SM, whole waves and a remainder; in each, one
# state in 32, some, most and all of a tile's; temperatures beyond either end,
# subnormal fractions, and products of tiny ones
@pytest.mark.parametrize("name,n", [("small", 515), ("small", 70000), ("gri53", 97),
                                    ("gri53", 4000), ("gri53", 456 * 32 + 7),
                                    ("large561", 64), ("large561", 153 * 32 + 5)])
def test_any_share_of_states_outside(name, n, synth_mech):
    from create_rate_subs_gb300.rates import RateSubs
    mech = synth_mech(name)
    N = mech.n_species
    T, P, Y = synth.make_states(N, n, seed=n + N)
    share = (np.arange(n) // 32) % 6  # by tile
    pick = np.zeros(n, bool)
    rng = np.random.default_rng(n)
    for k, p in enumerate((0.0, 1 / 32, 0.2, 0.6, 1.0, 0.0)):
        pick |= (share == k) & (rng.random(n) < p)
    pick[share == 1] = np.arange(n)[share == 1] % 32 == 5
    kind = (np.arange(n) // 192) % 3
    T[pick & (kind == 0)] = 195.0
    T[pick & (kind == 1)] = 6100.0
    Y[0, pick & (kind == 2)] = 5e-310
    tiny = share == 5
    Y[1:N - 1:3, tiny] = 1e-150
    ref = Oracle(mech.blob).eval(T, P, Y)
    G = gross_scale(mech.tables, ref["fwd"], ref["rev"], ref["pm"])
    rs = RateSubs(mech)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    w = rs.wdot(*d, mode="fp64").cpu().numpy()
    fin = np.all(np.isfinite(ref["wdot"]) & np.isfinite(G), axis=0)
    assert np.array_equal(np.all(np.isfinite(w), axis=0), fin)
    assert wdot_errors(w[:, fin], ref["wdot"][:, fin], G[:, fin])["scaled"] <= 1e-12
    # a state's bits depend neither on its neighbours nor on the launch
    some = np.flatnonzero(pick)[:: max(1, int(pick.sum()) // 40)]
    alone = rs.wdot(*[t[..., torch.from_numpy(some).cuda()].contiguous() for t in d], mode="fp64")
    assert np.array_equal(alone.cpu().numpy(), w[:, some], equal_nan=True)
