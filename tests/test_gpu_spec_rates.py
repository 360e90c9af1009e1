"""The batched eval_spec_rates by species (small batches) and in place (large
ones): the same operations in the same order, so the same bits."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", ["small", "gri53", "features"])
def test_both_layouts_give_the_same_bits(name, golden, synth_mech):
    from create_rate_subs_gb300.rates import RateSubs
    rs = RateSubs(golden(name)[0] if name == "features" else synth_mech(name))
    g = torch.Generator(device="cuda").manual_seed(1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = sms * 6 * 128  # states: the last batch by species
    rand = lambda rows: torch.randn((rows, line + 33), generator=g, dtype=torch.float64,
                                    device="cuda")
    fwd, rev, pm = rand(rs.n_reactions), rand(rs.n_rev), rand(max(rs.n_pdep, 1))
    large = rs.eval_spec_rates(fwd, rev, pm)
    for a, b in ((0, line), (line, line + 33), (7, 8)):
        part = rs.eval_spec_rates(fwd[:, a:b], rev[:, a:b], pm[:, a:b])
        assert torch.equal(part, large[:, a:b])
