"""The triangle attention core alone (px_triatt_flash) against fp64 at the edges of its tiles: 64 keys a work item of which the pair
bias of the first 32 reaches the logits by a copy into tensor memory and that of the others by addition, 128 queries and six rows a CTA."""
import pytest
import torch

from protenix_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [1, 7, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 161, 193])
def test_attention_core(n, masked):
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ldt, ldm = ops.ld(n), (n + 127) // 128 * 128
    q, k = (0.3 * draw(n, 4, n, 32)).half(), draw(n, 4, n, 32).half()
    v = torch.zeros(n, 4, 32, ldt, dtype=torch.half, device="cuda")
    v[..., :n] = draw(n, 4, 32, n).half()
    bias = torch.zeros(4, n, ldm, device="cuda")
    bias[..., :n] = 4 * draw(4, n, n)                         # far beyond what 16 bits would carry to the tolerance below
    bias[..., :n] += torch.linspace(-20, 20, n, device="cuda")[:, None]
    mb = torch.full((n, ldm), -float("inf"), device="cuda")
    mb[:, :n] = 0
    if masked:
        mb[:, :n][torch.rand(n, n, generator=g, device="cuda") < 0.3] = -1.44e9
    o = ops.triatt_flash(q, k, v, bias, mb)
    ops.device_error_flags()
    # the logits as fp32 holds them: a masked key's is -1.44e9 whatever was added before
    s = torch.einsum("uhqd,uhkd->uhqk", q.double(), k.double()) + bias[..., :n].double()
    s = (s.float() + mb[:, None, None, :n]).double()
    want = torch.einsum("uhqk,uhdk->uqhd", torch.softmax(s * 0.6931471805599453, -1), v[..., :n].double()).reshape(n, n, 128)
    assert torch.isfinite(o).all()
    rel = float((o.double() - want).norm() / want.norm())
    # P and o are rounded to fp16 (2^-12 each on average half of it), exponentials to 7.5e-5
    assert rel < 6e-4, rel


def test_attention_core_is_the_same_every_time():
    """Tiles handed back too early show as a wrong row in some of many runs."""
    n = 600
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k, v = (0.3 * draw(n, 4, n, 32)).half(), draw(n, 4, n, 32).half(), draw(n, 4, 32, n).half()
    ldm = (n + 127) // 128 * 128
    bias, mb = torch.zeros(4, n, ldm, device="cuda"), torch.full((n, ldm), -float("inf"), device="cuda")
    bias[..., :n] = 2 * draw(4, n, n)
    mb[:, :n] = 0
    first = ops.triatt_flash(q, k, v, bias, mb)
    differs = sum((ops.triatt_flash(q, k, v, bias, mb) != first).any() for _ in range(300))
    assert int(differs) == 0


@pytest.mark.parametrize("n_u", [1, 3, 4, 9, 100, 111, 114, 130])
def test_rows_do_not_depend_on_how_they_are_dealt_out(n_u):
    """CTAs of six rows, of three in the last wave, none for rows beyond the last: a slab of rows gives the bits of the whole."""
    n = 150
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k = (0.3 * draw(n, 4, n, 32)).half(), draw(n, 4, n, 32).half()
    v = torch.zeros(n, 4, 32, ops.ld(n), dtype=torch.half, device="cuda")
    v[..., :n] = draw(n, 4, 32, n).half()
    ldm = (n + 127) // 128 * 128
    bias, mb = torch.zeros(4, n, ldm, device="cuda"), torch.full((n, ldm), -float("inf"), device="cuda")
    bias[..., :n] = 2 * draw(4, n, n)
    mb[:, :n] = 0
    whole = ops.triatt_flash(q, k, v, bias, mb)
    for first in {0, (n - n_u) // 2, n - n_u}:
        rows = slice(first, first + n_u)
        part = ops.triatt_flash(q[rows].contiguous(), k[rows].contiguous(), v[rows].contiguous(), bias, mb[rows].contiguous())
        assert torch.equal(part, whole[rows])
    ops.device_error_flags()


def test_many_units_a_cta_equal_one(n=130):
    """Beyond forty units an SM a CTA has one unit, below it several; the rows are the same to the bit."""
    n_u = 6 * (41 * torch.cuda.get_device_properties(0).multi_processor_count // 8)
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k = (0.3 * draw(n_u, 4, n, 32)).half(), draw(n_u, 4, n, 32).half()
    v = torch.zeros(n_u, 4, 32, ops.ld(n), dtype=torch.half, device="cuda")
    v[..., :n] = draw(n_u, 4, 32, n).half()
    ldm = (n + 127) // 128 * 128
    bias, mb = torch.zeros(4, n, ldm, device="cuda"), torch.full((n_u, ldm), -float("inf"), device="cuda")
    bias[..., :n] = 2 * draw(4, n, n)
    mb[:, :n] = 0
    whole = ops.triatt_flash(q, k, v, bias, mb)
    for rows in (slice(0, 700), slice(n_u - 401, n_u)):
        assert torch.equal(ops.triatt_flash(q[rows], k[rows], v[rows], bias, mb[rows]), whole[rows])
    ops.device_error_flags()


@pytest.mark.parametrize("n_u, n", [(2400, 130), (40, 1000), (36, 1024)])
def test_several_units_a_cta_equal_one(n_u, n):
    """Up to 1024 keys CTAs work on several units where there are more units than SMs; a few rows have a CTA for each of theirs.  Same bits."""
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k = (0.3 * draw(n_u, 4, n, 32)).half(), draw(n_u, 4, n, 32).half()
    v = torch.zeros(n_u, 4, 32, ops.ld(n), dtype=torch.half, device="cuda")
    v[..., :n] = draw(n_u, 4, 32, n).half()
    ldm = (n + 127) // 128 * 128
    bias, mb = torch.zeros(4, n, ldm, device="cuda"), torch.full((n_u, ldm), -float("inf"), device="cuda")
    bias[..., :n] = 2 * draw(4, n, n)
    mb[:, :n] = -1.4e9 * (torch.rand(n_u, n, generator=g, device="cuda") < 0.1)
    whole = ops.triatt_flash(q, k, v, bias, mb)
    for first in (0, n_u // 2, n_u - 12):
        rows = slice(first, first + 12)
        assert torch.equal(ops.triatt_flash(q[rows], k[rows], v[rows], bias, mb[rows]), whole[rows])
    ops.device_error_flags()
