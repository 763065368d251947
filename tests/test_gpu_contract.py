"""The contraction alone and paired (one or two CTAs to a tile) at the edges of its tiles, against fp64 of the same operands.

Pairs take many tiles (two to an SM) of long contractions: with 128-byte lines from six row tiles and k = 448 on, with 32-byte sectors from k = 272,
with rows that straddle sectors from four row tiles and k = 152.  The last two sizes run in more CTAs than end evenly, so that each gets
ragged and whole tiles."""
import pytest
import torch

from protenix_b200 import _lib, ops

pytestmark = pytest.mark.gpu
SCALE = 2.0 ** -6


def _close(got, want):
    assert float((got.double() - want).norm()) < 5e-4 * float(want.norm()) + 1e-12


@pytest.mark.parametrize("channels,n", [(3, 1), (5, 64), (150, 100), (3, 129), (2, 200), (80, 256), (2, 257), (2, 385), (1, 512), (2, 520), (1, 777),
                                        (50, 384), (50, 390), (50, 400), (40, 520), (32, 640), (25, 641), (25, 777), (10, 1030),
                                        (128, 300), (128, 530)])
def test_contract(channels, n):
    torch.manual_seed(n)
    ld = ops.ld(n)
    a, b = (torch.zeros(channels, n, ld, device="cuda", dtype=torch.half) for _ in range(2))
    a[..., :n], b[..., :n] = torch.randn(2, channels, n, n, device="cuda").half()
    x = ops.trimul_contract(a, b)
    ops.device_error_flags()
    assert (x[..., n:] == 0).all()
    _close(x, SCALE * torch.nn.functional.pad(a.double() @ b.double().transpose(1, 2), (0, ld - n)))
    assert torch.equal(x, ops.trimul_contract(a, b))


@pytest.mark.parametrize("rows_a,rows_b,k", [(32, 96, 8), (160, 32, 72), (288, 544, 64), (544, 288, 136), (1024, 2080, 200),
                                           (3200, 3200, 144), (3200, 3232, 152), (3232, 3200, 272), (3264, 3200, 256),
                                           (3360, 3232, 448), (4096, 1056, 1000), (700 * 32, 32, 600)])
def test_outer(rows_a, rows_b, k):
    torch.manual_seed(k)
    a, b = torch.randn(rows_a, k, device="cuda").half(), torch.randn(rows_b, k, device="cuda").half()
    x = torch.full((rows_a, rows_b), float("nan"), device="cuda", dtype=torch.half)
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().px_opm_outer(a.data_ptr(), b.data_ptr(), x.data_ptr(), rows_a, rows_b, k, st), "px_opm_outer")
    ops.device_error_flags()
    _close(x, SCALE * (a.double() @ b.double().t()))
