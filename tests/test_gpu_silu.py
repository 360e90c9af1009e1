"""The SiLU of the fused network kernel (crs_mlp_infer), seen through two
identity layers, against FP64 over the whole range of bf16 inputs.

Tolerance: two approximations of 2^-22 and 2^-23 and the exponent's rounding, 4e-6
of the result in all; the activation is then rounded to bf16, so that it lies
between the roundings of the ends of that interval.  Where the reciprocal is below
2^-126 the result is zero, 2^-118 off at most.
"""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_silu_of_every_bf16():
    from create_rate_subs_gb300.surrogate import MLP
    bits = torch.arange(65536, dtype=torch.int32).to(torch.int16)
    z = bits.view(torch.bfloat16)
    z = z[torch.isfinite(z)]
    # the ends of the exponential's range in steps of a unit of bf16 are among them;
    # pad to rows of 64
    n = (z.numel() + 63) // 64
    x = torch.zeros(n * 64, dtype=torch.bfloat16)
    x[: z.numel()] = z
    net = MLP([64, 64, 64], seed=1)
    assert net.fused_ok()
    for layer in range(2):
        net.W[layer].zero_()
        net.W[layer][:64, :64] = torch.eye(64, device="cuda").to(torch.bfloat16)
        net.b32[layer].zero_()
    M = (n + 127) // 128 * 128
    X = torch.zeros(M, 64, dtype=torch.bfloat16, device="cuda")
    X[:n] = x.view(n, 64).cuda()
    # (one element per row: a sum with the other columns' huge or infinite products
    # would not be the element)
    out = torch.zeros(M, 64, device="cuda")
    got = torch.empty(n, 64, dtype=torch.float64)
    for c in range(64):
        one = torch.zeros_like(X)
        one[:, c] = X[:, c]
        net.infer(one, n, out)
        got[:, c] = out[:n, c].cpu().double()
    v = x.view(n, 64).double()
    want = v * torch.sigmoid(v)
    a = (want * (1 - 4e-6)).float().to(torch.bfloat16).double()
    b = (want * (1 + 4e-6)).float().to(torch.bfloat16).double()
    off = torch.maximum(torch.minimum(a, b) - got, got - torch.maximum(a, b))
    assert bool(torch.all(off <= 2.0 ** -118))
