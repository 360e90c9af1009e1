"""Fall-off centres of any size in the FP64 state tiles (crs_fx.cu): the
centre's sum keeps its relative accuracy, whatever its order of magnitude.

Tolerance: the FP64 modes' gross-rate scaled error of 1e-12.
"""
import numpy as np
import pytest

from create_rate_subs_gb300 import synth
from oracle.oracle import Oracle, gross_scale, wdot_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# centres of exp(-T / 100), 5e-4 to 1e-12 over the range, of one, two and three
# terms; one beside a term that is zero; a difference of two terms, which
# changes its sign at 2008 K (no states within 20 K, where the terms cancel to
# less than 1/400); SRI bases as small
@pytest.mark.parametrize("form", ["TROE / 1. 100. 100. /", "TROE / 0.5 100. 100. /",
                                  "TROE / 0.3 90. 110. 25000. /", "TROE / 0.999999 1.E-30 100. /",
                                  "TROE / 5.0 1000. 900. /", "SRI / 1.E-5 100. 90. /",
                                  "SRI / 0.4 20000. 80. 1.5 0.2 /"])
def test_small_centres(form, tmp_path):
    from create_rate_subs_gb300.mechanism import Mechanism
    from create_rate_subs_gb300.rates import RateSubs
    text, therm = synth.make_mechanism(**synth.CONFIGS["small"])
    lines = ["    " + form if "TROE" in line else line for line in text.split("\n")]
    assert sum(form in line for line in lines) == 3
    mp, tp = tmp_path / "mech.inp", tmp_path / "therm.dat"
    mp.write_text("\n".join(lines))
    tp.write_text(therm)
    mech = Mechanism.from_chemkin(str(mp), str(tp))
    N = mech.n_species
    T, P, Y = synth.make_states(N, 4099, seed=N, p_atm=(1e-3, 1e3))
    T[np.abs(T - 2008.3) < 20.0] = 900.0
    ref = Oracle(mech.blob).eval(T, P, Y)
    G = gross_scale(mech.tables, ref["fwd"], ref["rev"], ref["pm"])
    rs = RateSubs(mech)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    w = rs.wdot(*d, mode="fp64").cpu().numpy()
    assert wdot_errors(w, ref["wdot"], G)["scaled"] <= 1e-12
    assert rs.status() == (0, 0)


def test_absent_reactants_and_colliders(tmp_path):
    """Rates with up to four absent reactants, with very small constants, and
    fall-off rates without their collider are zero, as in the general code."""
    from create_rate_subs_gb300.mechanism import Mechanism
    from create_rate_subs_gb300.rates import RateSubs
    text, therm = synth.make_mechanism(**synth.CONFIGS["small"])
    text = text[: text.rindex("END")] + """2H+2HO<=>2H2O 1.0E-200 -5.0 150000.0
2H+2HO=>2H2O 1.0E+40 3.0 0.0
H+HO(+H2O)<=>H2O(+H2O) 1.0E+13 0.0 0.0
   LOW / 1.0E+18 -1.0 0.0 /
   TROE / 0.5 100. 1000. /
2HO(+O2)<=>H2O+O(+O2) 1.0E+13 0.0 0.0
   HIGH / 1.0E+15 0.5 20.0 /
   SRI / 0.5 300.0 900.0 1.2 0.3 /
END
"""
    mp, tp = tmp_path / "mech.inp", tmp_path / "therm.dat"
    mp.write_text(text)
    tp.write_text(therm)
    mech = Mechanism.from_chemkin(str(mp), str(tp))
    N = mech.n_species
    T, P, Y = synth.make_states(N, 515, seed=N, t_range=(250.0, 3000.0), p_atm=(1e-6, 1e3))
    at = {k: list(mech.names).index(k) for k in ("H", "HO", "H2O", "O2")}
    Y[at["H"], 0::3] = 0.0
    Y[at["HO"], 0::6] = 0.0
    Y[at["H2O"], 1::3] = 0.0
    Y[at["H2O"], 0::6] = 0.0
    Y[at["O2"], 2::6] = 0.0
    ref = Oracle(mech.blob).eval(T, P, Y)
    G = gross_scale(mech.tables, ref["fwd"], ref["rev"], ref["pm"])
    rs = RateSubs(mech)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
    w = rs.wdot(*d, mode="fp64").cpu().numpy()
    assert np.all(w[G == 0.0] == 0.0)
    assert wdot_errors(w, ref["wdot"], G)["scaled"] <= 1e-12
    assert rs.status() == (0, 0)
