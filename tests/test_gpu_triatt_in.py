"""The projections of the triangle attention (px_triatt_in_proj) against fp64 at the edges of its tiles and of the tiles per CTA, with the
mask bias and the padding of both bias tensors."""
import math

import pytest
import torch
import torch.nn.functional as F

from protenix_b200 import ops

pytestmark = pytest.mark.gpu
LOG2E = math.log2(math.e)


def inputs(n_u, n_t, dtype, ending):
    g = torch.Generator("cuda").manual_seed(1000 * n_u + n_t)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    shape = (n_t, n_u) if ending else (n_u, n_t)
    z = ((0.5 + draw(*shape, 128)) * (0.3 + draw(*shape, 1).abs())).to(dtype)
    mask = (torch.rand(*shape, generator=g, device="cuda") > 0.2).float()
    wt = torch.float16 if dtype == torch.float32 else dtype
    weights = [1 + 0.2 * draw(128), 0.2 * draw(128), (0.09 * draw(4, 128)).to(wt)] + [(0.09 * draw(128, 128)).to(wt) for _ in range(3)]
    return z, mask, weights


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("n_u,n_t", [(1, 1), (3, 127), (2, 128), (5, 129), (149, 130), (300, 257)])
def test_triatt_in(n_u, n_t, ending, dtype):
    z, mask, w = inputs(n_u, n_t, dtype, ending)
    q, k, v, bias, mb = ops.triatt_in_proj(z, mask, *w, ending=ending)
    ops.device_error_flags()
    y = z.double()
    rows, m = (y.transpose(0, 1), mask.T) if ending else (y, mask)
    d = [t.double() for t in w]
    y = F.layer_norm(rows, (128,), d[0], d[1], 1e-5)
    heads = lambda t: (y @ t.T).view(n_u, n_t, 4, 32).permute(0, 2, 1, 3)
    want = (heads(d[3]) * LOG2E / math.sqrt(32), heads(d[4]), heads(d[5]).transpose(2, 3), (y @ d[2].T).permute(2, 0, 1) * LOG2E)
    # folded weights and standardised rows of 11 bits (3e-4 each) and the rounding of q, k, v (3e-4); bf16: folded weights of 8 bits
    tol = 1e-3 if dtype == torch.float32 else 3e-3
    for name, got, ref in zip("qkvb", (q, k, v[..., :n_t], bias[..., :n_t]), want):
        rel = float((got.double() - ref).norm() / ref.norm())
        assert rel < tol, (name, rel)
    # the mask bias is exact for masks of zeros and ones
    assert torch.equal(mb[:, :n_t], torch.where(m > 0, 0.0, torch.tensor(-1e9, device="cuda") * torch.tensor(LOG2E, device="cuda")))
    assert bool((mb[:, n_t:] == -math.inf).all()) and not bool(bias[..., n_t:].any()) and not bool(v[..., n_t:].any())


@pytest.mark.parametrize("ending", [False, True])
def test_rows_beyond_l2_equal_a_slab(ending):
    """More rows than L2 holds are loaded with fewer tiles on their way; each u is computed by itself, so a slab of them gives the same
    bits."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    n_t = 500
    n_u = -(-(3 * l2 // 2) // (n_t * 256)) + 5
    z, mask, w = inputs(n_u, n_t, torch.float32, ending)
    whole = ops.triatt_in_proj(z, mask, *w, ending=ending)
    for u0 in (0, n_u // 2, n_u - 3):
        part = (slice(None), slice(u0, u0 + 3)) if ending else (slice(u0, u0 + 3),)
        slab = ops.triatt_in_proj(z[part].contiguous(), mask[part].contiguous(), *w, ending=ending)
        for name, a, b in zip("qkvbm", whole, slab):
            assert torch.equal(a[:, u0:u0 + 3] if name == "b" else a[u0:u0 + 3], b), name
    ops.device_error_flags()


@pytest.mark.parametrize("ending", [False, True])
def test_two_runs_a_tile_beyond_l2(ending, n_t=520):
    """As above where tiles are made of two runs of 64, and the same rows against fp64."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    n_u = -(-(3 * l2 // 2) // (n_t * 256)) + 5
    z, mask, w = inputs(n_u, n_t, torch.float32, ending)
    q, k, v, bias, mb = whole = ops.triatt_in_proj(z, mask, *w, ending=ending)
    for u0 in (0, n_u // 2, n_u - 3):
        part = (slice(None), slice(u0, u0 + 3)) if ending else (slice(u0, u0 + 3),)
        slab = ops.triatt_in_proj(z[part].contiguous(), mask[part].contiguous(), *w, ending=ending)
        for name, a, b in zip("qkvbm", whole, slab):
            assert torch.equal(a[:, u0:u0 + 3] if name == "b" else a[u0:u0 + 3], b), name
        rows = z[part].double().transpose(0, 1) if ending else z[part].double()
        d = [t.double() for t in w]
        y = F.layer_norm(rows, (128,), d[0], d[1], 1e-5)
        heads = lambda t: (y @ t.T).view(3, n_t, 4, 32).permute(0, 2, 1, 3)
        want = (heads(d[3]) * LOG2E / math.sqrt(32), heads(d[4]), heads(d[5]).transpose(2, 3), (y @ d[2].T).permute(2, 0, 1) * LOG2E)
        got = (q[u0:u0 + 3], k[u0:u0 + 3], v[u0:u0 + 3, ..., :n_t], bias[:, u0:u0 + 3, :n_t])
        for name, a, b in zip("qkvb", got, want):      # the tolerance of test_triatt_in
            assert float((a.double() - b).norm() / b.norm()) < 1e-3, name
    assert bool((mb[:, n_t:] == -math.inf).all()) and not bool(bias[..., n_t:].any()) and not bool(v[..., n_t:].any())
    ops.device_error_flags()


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("n_t", [384, 400])
def test_any_number_of_tiles_a_cta_gives_the_same_bits(ending, n_t):
    """bf16 rows are measured by one set of warps or by two, by the tiles of a CTA: many, some and one of them here."""
    z, mask, w = inputs(n_t, n_t, torch.bfloat16, ending)
    whole = ops.triatt_in_proj(z, mask, *w, ending=ending)
    for n_u in (300, 100, 37, 10, 1):
        part = (slice(None), slice(7, 7 + n_u)) if ending else (slice(7, 7 + n_u),)
        slab = ops.triatt_in_proj(z[part].contiguous(), mask[part].contiguous(), *w, ending=ending)
        for name, a, b in zip("qkvbm", whole, slab):
            assert torch.equal(a[:, 7:7 + n_u] if name == "b" else a[7:7 + n_u], b), (name, n_u)
    ops.device_error_flags()
