"""The FP64 work that the state tiles keep, counted by hand on the 10-species
mechanism (CPU): 27 reversible reactions with 85 nonzero net coefficients, five
three-body and three fall-off ones with 30 efficiencies."""
from create_rate_subs_gb300 import work


def test_hand_counts(synth_mech):
    t = synth_mech("small").tables
    fixed = work.fp64_slots(t, "fixed", 9.0)
    # two sums over 10 species, 30 efficiencies, two products for each of the five
    # three-body reactions, 27 differences, 85 terms
    assert fixed["parts"] == {"mass_fraction_sums": 20, "third_body": 30 + 10, "net_rate": 27,
                              "accumulation": 85}
    assert fixed["slots"] == 172
    # 27 differences, 8 products with a pressure modification
    operand = work.fp64_slots(t, "operand", 9.0)
    assert operand["parts"] == {"net_rate": 27, "pres_mod_product": 8}
    mixed = work.fp64_slots(t, "mixed", 9.0)
    assert mixed["slots"] == operand["slots"] + 85 == 120
