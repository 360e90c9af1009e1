"""crs_surrogate_output2 and crs_surrogate_disagreement over numbers of species
and of states, against the same formulas in PyTorch, and from several threads.

Tolerances: expm1 and its products in fp32 (4 units of 2^-24, the exponent's
rounding |y| 2^-24 on top, |y| < 8); sums of nsp terms in fp32; a bf16 input
half a unit of 2^-8.
"""
import ctypes
import threading

import pytest

from create_rate_subs_gb300 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

NELEM = 3


class Case(object):
    def __init__(self, n, nsp, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rand = lambda *s: torch.randn(s, generator=g, device="cuda")
        self.n, self.nsp, self.ldy = n, nsp, nsp + 3
        self.Ya = rand(n, self.ldy)
        self.Yb = self.Ya + 0.1 * rand(n, self.ldy)
        self.sm = 1.0 + torch.rand(max(nsp, 1), generator=g, device="cuda")
        self.se = torch.randint(-60, 60, (max(nsp, 1),), generator=g, device="cuda",
                                dtype=torch.int32)
        self.cons = torch.rand((NELEM, max(nsp, 1)), generator=g, device="cuda")
        self.est = rand(n, 2)
        self.box = (torch.rand(n, generator=g, device="cuda") < 0.1).to(torch.uint8)
        self.w = torch.full((max(nsp, 1), n), -7.0, dtype=torch.float64, device="cuda")
        self.fb = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
        self.gate = torch.full((n,), -7.0, device="cuda")
        self.X = torch.zeros(n, 64, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()

    def run(self, stream):
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        lib, s = _lib.load(), ctypes.c_void_p(stream)
        _lib.check(lib.crs_surrogate_output2(
            self.n, p(self.Ya), p(self.Yb), self.ldy, self.nsp, p(self.sm), p(self.se),
            p(self.cons), NELEM, 0.5, 0.7, p(self.est), 2, 0.4, p(self.box), p(self.w), self.n,
            p(self.fb), p(self.gate), s))
        _lib.check(lib.crs_surrogate_disagreement(self.n, p(self.Ya), p(self.Yb), self.ldy,
                                                  self.nsp, -1.0, 0.5, p(self.X), 64, 5, s))

    def check(self):
        k = self.nsp
        ya, yb = self.Ya[:, :k], self.Yb[:, :k]
        y = (0.5 * (ya + yb)).double()
        u = torch.sign(y) * torch.expm1(y.abs())
        want = (u * self.sm[:k].double() * torch.exp2(self.se[:k].double())).t()
        assert bool(torch.all((self.w[:k] - want).abs() <= 16 * 2.0 ** -24 * want.abs()))
        d = (ya - yb).abs().amax(dim=1) if k else torch.zeros(self.n, device="cuda")
        ld = torch.log10(d + 1e-4)
        gate = 0.7 * ld + self.est[:, 0]
        assert bool(torch.all((self.gate - gate).abs() <= 8 * 2.0 ** -24 * (4 + gate.abs())))
        want = (ld + 1.0) / 0.5
        assert bool(torch.all((self.X[:, 5].float() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5))
        c = self.cons[:, :k].double().t()
        worst = ((u @ c).abs() / ((u.abs() + 1.0) @ c + (k == 0))).amax(dim=1)
        fb = (worst > 0.5) | (gate > 0.4) | (self.box != 0)
        # a state within rounding of a threshold may go either way
        near = ((worst - 0.5).abs() <= (k + 32) * 2.0 ** -24) | ((gate - 0.4).abs() <= 1e-5)
        assert bool(torch.all((self.fb.bool() == fb) | near))


def test_threads_with_different_sizes():
    """Each call's launch has the shared memory that it asks for, whatever other
    threads ask for at the same time."""
    cases = [Case(257, nsp, nsp) for nsp in (53, 64, 96, 40)]
    errors = []

    def work(c):
        try:
            torch.cuda.set_device(0)
            s = torch.cuda.Stream()
            for _ in range(400):
                c.run(s.cuda_stream)
            s.synchronize()
        except Exception as e:  # reported by the test
            errors.append(e)
    threads = [threading.Thread(target=work, args=(c,)) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for c in cases:
        c.check()


# rows by threads and by warps, their lines at 32, 48 and 97 species and at one
# CTA per SM; fewer than eight warps; species that no column of means holds; none
@pytest.mark.parametrize("n,nsp", [(1, 1), (33, 0), (1000, 10), (77, 31), (77, 47), (77, 48),
                                   (32767, 33), (32768, 33), (4099, 96), (4099, 101),
                                   (4099, 194), (40000, 194), (65, 1551), (4099, 1551),
                                   (300, 1552), (300, 2001)])
def test_sizes(n, nsp):
    c = Case(n, nsp, n + nsp)
    c.run(torch.cuda.current_stream().cuda_stream)
    c.check()
