"""The output stage of the triangle multiplication (px_trimul_out) against fp64 at the edges of its tiles and of the tiles per CTA, with
rows of x near zero mean and far from it: their statistics are summed across the tile in shared memory."""
import pytest
import torch
import torch.nn.functional as F

from protenix_b200 import ops

pytestmark = pytest.mark.gpu


def errors(n_i, n_j, dtype, shift):
    """Relative errors of the update (fp32 rows) or of the result (bf16 rows)."""
    g = torch.Generator("cuda").manual_seed(1000 * n_i + n_j)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    z = (0.5 + draw(n_i, n_j, 128)).to(dtype)
    x = 7.0 * torch.ones(128, n_i, ops.ld(n_j), device="cuda")
    x[:, :, :n_j] = (shift + draw(128, n_i, n_j)) * (0.3 + draw(1, n_i, n_j).abs())
    x = x.half()
    w_in, b_in, w_out, b_out = 1 + 0.2 * draw(128), 0.2 * draw(128), 1 + 0.2 * draw(128), 0.2 * draw(128)
    w_z, w_g = (0.09 * draw(128, 128)).half(), (0.09 * draw(128, 128)).to(torch.float16 if dtype == torch.float32 else dtype)
    d = lambda t: t.double()
    rows = d(x[:, :, :n_j]).permute(1, 2, 0) * 64.0            # x is stored times 1/64
    update = (F.layer_norm(rows, (128,), d(w_out), d(b_out), 1e-5) @ d(w_z).T) * torch.sigmoid(
        F.layer_norm(d(z), (128,), d(w_in), d(b_in), 1e-5) @ d(w_g).T)
    out = ops.trimul_out(x, z.clone(), w_in, b_in, w_out, b_out, w_z, w_g)
    ops.device_error_flags()
    want = update if dtype == torch.float32 else d(z) + update
    got = d(out) - d(z) if dtype == torch.float32 else d(out)
    return float((got - want).norm() / want.norm())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_i,n_j", [(1, 1), (3, 127), (2, 128), (5, 129), (149, 130), (300, 257)])
def test_trimul_out(n_i, n_j, dtype):
    # fp32 rows: folded weights and gate operands of 11 bits (3e-4 each), the approximate tanh (5e-4); bf16 rows: the rounding of the
    # result (2^-9 / sqrt 3) and of the folded gate weights.  Far from zero mean the correction step's 17 bits weigh 30 times as much.
    tol = 1e-3 if dtype == torch.float32 else 3e-3
    for shift in (0.2, 30.0):
        rel = errors(n_i, n_j, dtype, shift)
        assert rel < tol, (rel, shift)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_i,n_j", [(1, 8), (2, 72), (3, 40), (75, 120), (149, 136)])
def test_trimul_out_across_rows(n_i, n_j, dtype):
    """Without pad columns the tiles run on from row to row (the tolerances are those of test_trimul_out)."""
    for shift in (0.2, 30.0):
        rel = errors(n_i, n_j, dtype, shift)
        assert rel < (1e-3 if dtype == torch.float32 else 3e-3), (rel, shift)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [64, 100, 136, 150, 200, 448, 520])
def test_tiles_are_cut_in_three_ways_with_the_same_bits(n, dtype):
    """Rows by themselves, runs of 64 and one row, by the number of tiles; a few rows of the whole are cut in another way or lie elsewhere in it."""
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    z, x = draw(n, n, 128).to(dtype), torch.zeros(128, n, ops.ld(n), dtype=torch.half, device="cuda")
    x[..., :n] = draw(128, n, n).half()
    wt = torch.float16 if dtype == torch.float32 else dtype
    vectors = [1 + 0.2 * draw(128), 0.2 * draw(128), 1 + 0.2 * draw(128), 0.2 * draw(128)]
    o, w_z, w_g = draw(n, n, 128).half(), (0.09 * draw(128, 128)).half(), (0.09 * draw(128, 128)).to(wt)
    mul = ops.trimul_out(x, z.clone(), *vectors, w_z, w_g)
    start = ops.triatt_out(o, z.clone(), *vectors[:2], w_g, w_z)
    end = ops.triatt_out(o, z.clone(), *vectors[:2], w_g, w_z, ending=True)
    for n_u in (1, 7, 40, n - 3):
        rows = slice(n - n_u, n)
        part = z[rows].clone()
        assert torch.equal(ops.trimul_out(x[:, rows].contiguous(), part.clone(), *vectors, w_z, w_g), mul[rows])
        assert torch.equal(ops.triatt_out(o[rows], part, *vectors[:2], w_g, w_z), start[rows])
        part = z[:, rows].contiguous()
        assert torch.equal(ops.triatt_out(o[rows], part, *vectors[:2], w_g, w_z, ending=True), end[:, rows])
    ops.device_error_flags()


@pytest.mark.parametrize("ending", [False, True])
@pytest.mark.parametrize("n", [64, 150, 200, 520])
def test_update_alone_is_what_is_added(n, ending):
    """The form that writes the update in fp16 from standardised rows, in the cuts that it takes, against the one that adds it to an fp32 z."""
    g = torch.Generator("cuda").manual_seed(n)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    z, o = draw(n, n, 128), draw(n, n, 128).half()
    zn = ops.standardise_rows(z)
    args = 1 + 0.2 * draw(128), 0.2 * draw(128), (0.09 * draw(128, 128)).half(), (0.09 * draw(128, 128)).half()
    update = ops.triatt_out(o, zn, *args, ending=ending)
    added = ops.triatt_out(o, z.clone(), *args, ending=ending, zn=zn).double() - z.double()
    # rounding to fp16, 2^-11 / sqrt 3 at most on average; the sum's own rounding is far below
    assert float((update.double() - added).norm() / added.norm()) < 4e-4
    ops.device_error_flags()
