"""crs_mlp_row_sums of short rows and of many rows (a warp per row), on both
sides of the lines to a CTA per row, 2,048 columns and 1,024 rows: the sums are
formed in one order, so a row's bits are the same wherever it is formed.  The
sum of m terms in fp32, 32 chains and five more additions: within
(m / 32 + 6) 2^-24 of the terms' magnitudes."""
import ctypes

import pytest

from create_rate_subs_gb300 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _sums(x, rows, m):
    out = torch.full((rows,), 7.0, device="cuda")
    _lib.check(_lib.load().crs_mlp_row_sums(
        ctypes.c_void_p(x.data_ptr()), x.stride(0), rows, m, ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return out


@pytest.mark.parametrize("rows,m,ld", [(1, 1, 1), (9, 31, 33), (1025, 128, 128), (3, 2048, 2056),
                                       (1024, 2049, 2049), (1025, 2049, 2050), (1030, 4097, 4104)])
def test_row_sums(rows, m, ld):
    g = torch.Generator(device="cuda").manual_seed(rows + m)
    x = torch.randn((rows, ld), generator=g, device="cuda").to(torch.bfloat16)
    out = _sums(x, rows, m)
    v = x[:, :m].double()
    tol = (m / 32 + 6) * 2.0 ** -24 * v.abs().sum(dim=1)
    assert bool(torch.all((out.double() - v.sum(dim=1)).abs() <= tol))
    few = min(rows, 5)
    assert torch.equal(_sums(x, few, m), out[:few])
