"""crs_mlp_row_sums at the edges of its chunks of 4,096 columns and with rows
that no 16-byte load may start on.  The sum of m terms in fp32, 32 chains and
five more additions: within (m / 32 + 6) 2^-24 of the terms' magnitudes."""
import ctypes

import pytest

from create_rate_subs_gb300 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,m,ld", [(1, 1, 1), (3, 31, 33), (5, 4096, 4096), (2, 4097, 4104),
                                       (7, 8191, 8191), (53, 16384, 16384)])
def test_row_sums(rows, m, ld):
    g = torch.Generator(device="cuda").manual_seed(rows + m)
    x = torch.randn((rows, ld), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((rows,), 7.0, device="cuda")
    _lib.check(_lib.load().crs_mlp_row_sums(
        ctypes.c_void_p(x.data_ptr()), ld, rows, m, ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    v = x[:, :m].double()
    tol = (m / 32 + 6) * 2.0 ** -24 * v.abs().sum(dim=1)
    assert bool(torch.all((out.double() - v.sum(dim=1)).abs() <= tol))
