"""The projections of the triangle multiplication (px_trimul_in_proj) against fp64 at the edges of its tiles and of the tiles per CTA, rows
far from zero mean among them, and the same bits from call to call (the statistics of bf16 rows are two tiles' at a time)."""
import pytest
import torch
import torch.nn.functional as F

from protenix_b200 import ops

pytestmark = pytest.mark.gpu


def inputs(n_u, n_t, dtype, incoming):
    g = torch.Generator("cuda").manual_seed(1000 * n_u + n_t)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    shape = (n_t, n_u) if incoming else (n_u, n_t)
    z = ((0.5 + draw(*shape, 128)) * (0.3 + draw(*shape, 1).abs()) + draw(*shape, 1)).to(dtype)
    mask = (torch.rand(*shape, generator=g, device="cuda") > 0.2).float()
    wt = torch.float16 if dtype == torch.float32 else dtype
    return z, mask, [1 + 0.2 * draw(128), 0.2 * draw(128)] + [(0.09 * draw(128, 128)).to(wt) for _ in range(4)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("incoming", [False, True])
@pytest.mark.parametrize("n_u,n_t", [(1, 1), (3, 64), (3, 65), (2, 127), (2, 128), (5, 129), (75, 120), (300, 193)])
def test_trimul_in(n_u, n_t, incoming, dtype):
    z, mask, w = inputs(n_u, n_t, dtype, incoming)
    a, b = ops.trimul_in_proj(z, mask, *w, incoming)
    ops.device_error_flags()
    y, m = z.double(), mask.double()[..., None]
    if incoming:
        y, m = y.transpose(0, 1), m.transpose(0, 1)
    d = [t.double() for t in w]
    y = F.layer_norm(y, (128,), d[0], d[1], 1e-5)
    # folded weights and standardised rows of 11 bits (3e-4 each), the rounding of the result and the tanh (3e-4 together); bf16: 8 bits
    tol = 1e-3 if dtype == torch.float32 else 4e-3
    for got, p, g in ((a, d[2], d[3]), (b, d[4], d[5])):
        want = (m * (y @ p.T) * torch.sigmoid(y @ g.T)).permute(2, 0, 1)
        assert float((got[..., :n_t].double() - want).norm() / want.norm().clamp_min(1e-9)) < tol
        assert not bool(got[..., n_t:].any())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_trimul_in_is_the_same_every_time(dtype):
    z, mask, w = inputs(700, 700, dtype, False)
    first = ops.trimul_in_proj(z, mask, *w, False)
    differs = 0
    for _ in range(100):
        again = ops.trimul_in_proj(z, mask, *w, False)
        differs += int(not (torch.equal(again[0], first[0]) and torch.equal(again[1], first[1])))
    assert differs == 0
    ops.device_error_flags()


@pytest.mark.parametrize("n", [8, 40, 136, 200])
def test_tiles_across_rows_equal_a_slab_of_one(n):
    """Without pad columns the tiles of the outgoing projection run on from row to row; a slab of one row has them by itself."""
    z, mask, w = inputs(n, n, torch.float32, False)
    a, b = ops.trimul_in_proj(z, mask, *w, False)
    for u in (0, n // 2, n - 1):
        pa, pb = ops.trimul_in_proj(z[u:u + 1].contiguous(), mask[u:u + 1].contiguous(), *w, False)
        assert torch.equal(pa[:, 0], a[:, u]) and torch.equal(pb[:, 0], b[:, u])
    ops.device_error_flags()


@pytest.mark.parametrize("n_u", [1, 2, 3, 75])
def test_ends_of_two_rows_share_a_tile(n_u):
    """130 t: two whole runs of 64 and a ragged one; the ends of neighbouring rows meet in one tile, the last row's may stand alone."""
    z, mask, w = inputs(76, 130, torch.bfloat16, False)
    a, b = ops.trimul_in_proj(z, mask, *w, False)
    pa, pb = ops.trimul_in_proj(z[:n_u].contiguous(), mask[:n_u].contiguous(), *w, False)
    assert torch.equal(pa, a[:, :n_u]) and torch.equal(pb, b[:, :n_u])
    ops.device_error_flags()
