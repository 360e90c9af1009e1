"""State tiles of mechanisms whose columns leave little shared memory: small
tables in global memory, then no room at all (crs_fx.cu, crs_mixed_tile.cu)."""
import numpy as np
import pytest

from create_rate_subs_gb300 import synth
from oracle.oracle import Oracle, gross_scale, wdot_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _with_inert_species(n):
    """The 561-species mechanism and n copies of argon."""
    text, therm = synth.make_mechanism(**synth.CONFIGS["large561"])
    lines = therm.split("\n")
    at = [k for k, line in enumerate(lines) if line.startswith("AR ")][0]
    entry = lines[at:at + 4]
    names = ["ZZ%dQ" % k for k in range(n)]
    for name in names:
        lines[-2:-2] = [name.ljust(18) + entry[0][18:]] + entry[1:]
    return text.replace("SPECIES\n", "SPECIES\n" + " ".join(names) + "\n"), "\n".join(lines)


# 720: small tables on chip; 741 and 760: in global memory; 791: other kernels
@pytest.mark.parametrize("species", [720, 741, 760, 791])
def test_species_to_the_end_of_shared_memory(species, tmp_path):
    from create_rate_subs_gb300.mechanism import Mechanism
    from create_rate_subs_gb300.rates import RateSubs
    text, therm = _with_inert_species(species - 561)
    (tmp_path / "m").write_text(text)
    (tmp_path / "t").write_text(therm)
    mech = Mechanism.from_chemkin(str(tmp_path / "m"), str(tmp_path / "t"))
    N = mech.n_species
    assert N == species
    rs = RateSubs(mech)
    for n in (33, 153 * 32 + 5):
        T, P, Y = synth.make_states(N, n, seed=n)
        T[3::50] = 6100.0
        ref = Oracle(mech.blob).eval(T, P, Y)
        G = gross_scale(mech.tables, ref["fwd"], ref["rev"], ref["pm"])
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (T, P, Y[: N - 1])]
        for mode, tol in (("fp64", 1e-12), ("mixed", 1e-6)):
            w = rs.wdot(*d, mode=mode).cpu().numpy()
            assert wdot_errors(w, ref["wdot"], G)["scaled"] <= tol
    assert rs.status() == (0, 0)
