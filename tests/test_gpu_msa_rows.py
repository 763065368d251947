"""The MSA embedding's kernels (values, gated output, transition, outer-product operands) through MSAStack and OuterProductMean:
no further from the modules' composition in fp64 than the same composition in fp32."""
import pytest
import torch
from torch.nn import functional as F

import protenix_b200 as px
from protenix_b200 import ops
from protenix_b200.init_utils import randomize_parameters_
from protenix_b200.msa import MSAStack

pytestmark = pytest.mark.gpu


def _stack(mod, m, w, dt):
    att, tr, g = mod.msa_pair_weighted_averaging, mod.transition_m, (lambda p: p.detach().to(dt))
    m, w = m.to(dt), w.to(dt)
    s, n, _ = m.shape
    x = F.layer_norm(m, (64,), g(att.layernorm_m.weight), g(att.layernorm_m.bias), att.layernorm_m.eps)
    v = F.linear(x, g(att.linear_no_bias_mv.weight)).view(s, n, 8, 8)
    o = torch.sigmoid(F.linear(x, g(att.linear_no_bias_mg.weight))) * torch.einsum("hij,sjhc->sihc", w, v).reshape(s, n, 64)
    m = m + F.linear(o, g(att.linear_no_bias_out.weight))
    y = F.layer_norm(m, (64,), g(tr.layernorm1.weight), g(tr.layernorm1.bias), tr.layernorm1.eps)
    h = F.silu(F.linear(y, g(tr.linear_no_bias_a.weight))) * F.linear(y, g(tr.linear_no_bias_b.weight))
    return m + F.linear(h, g(tr.linear_no_bias.weight))


@pytest.mark.parametrize("s,n,chunk", [(1, 1, 2048), (3, 17, 2048), (64, 33, 2048), (127, 40, 2048), (129, 24, 100), (130, 130, 64)])
def test_msa_stack(s, n, chunk):
    torch.manual_seed(s * n)
    mod = randomize_parameters_(MSAStack(msa_chunk_size=chunk), 3).cuda().eval()
    m, z = 2 * torch.randn(s, n, 64, device="cuda") + 0.5, torch.randn(n, n, 128, device="cuda")
    relf = lambda a, b: float((a.double() - b).norm() / b.norm())
    with torch.no_grad():
        w = mod.msa_pair_weighted_averaging.pair_weights(z)
        want = _stack(mod, m, w, torch.float64)
        single = relf(_stack(mod, m, w, torch.float32), want)
        got = mod(m.clone(), z)
        ops.device_error_flags()
        assert relf(got, want) < 2 * single + 1e-7, (relf(got, want), single)
        assert torch.equal(got, mod(m.clone(), z))


@pytest.mark.parametrize("s,n,masked", [(1, 1, False), (7, 5, True), (128, 9, True), (129, 3, False), (136, 20, True)])
def test_outer_product_operands(s, n, masked):
    """px_msa_opm_prep: values, zero padding and both halves of the projection."""
    torch.manual_seed(s)
    mod = randomize_parameters_(px.OuterProductMean(64, 128, 32), 5).cuda()
    m = torch.randn(s, n, 64, device="cuda")
    mask = (torch.rand(s, n, device="cuda") > 0.3).float() if masked else None
    ld = (s + 7) // 8 * 8
    a, b = (torch.full((n * 32, ld), 7.0, dtype=torch.float16, device="cuda") for _ in range(2))
    from protenix_b200 import _lib

    ln = mod.layer_norm
    p = lambda t: None if t is None else t.data_ptr()
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    w = torch.empty(lib.px_msa_rows_weights_bytes(), dtype=torch.uint8, device="cuda")
    _lib.check(lib.px_msa_rows_prepare(p(mod.linear_1.weight), p(mod.linear_2.weight), p(w), st), "px_msa_rows_prepare")
    _lib.check(lib.px_msa_opm_prep(p(m), p(mask), p(ln.weight), p(ln.bias), p(w), p(a), p(b), s, n, ld, ln.eps, st), "px_msa_opm_prep")
    x = F.layer_norm(m.double(), (64,), ln.weight.detach().double(), ln.bias.detach().double(), ln.eps)
    for got, lin in ((a, mod.linear_1), (b, mod.linear_2)):
        want = F.linear(x, lin.weight.detach().double()) * (1.0 if mask is None else mask.double()[..., None])
        want = want.permute(1, 2, 0).reshape(n * 32, s)
        assert (got[:, s:] == 0).all()
        assert float((got[:, :s].double() - want).abs().max()) < 6e-4 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("s,n", [(1, 1), (16, 64), (17, 65), (33, 129), (16, 200)])
def test_weighted_average(s, n):
    """px_msa_weights and px_msa_average at the edges of their tiles (128 rows, 64 keys, 16 sequences)."""
    from protenix_b200 import _lib

    torch.manual_seed(n)
    ld, lib, st = (n + 7) // 8 * 8, _lib.load(), torch.cuda.current_stream().cuda_stream
    logits, v = 3 * torch.randn(8, n, n, device="cuda"), torch.randn(8, n, s * 8, device="cuda")
    planes, rest = [], v.clone()
    for _ in range(3):
        planes.append(rest.bfloat16())
        rest -= planes[-1].float()
    vp = torch.stack(planes, 1).contiguous()
    wp = torch.empty(8, 3, n, ld, dtype=torch.bfloat16, device="cuda")
    got = torch.full((8, n, s * 8), float("nan"), device="cuda")
    _lib.check(lib.px_msa_weights(logits.data_ptr(), wp.data_ptr(), n, ld, st), "px_msa_weights")
    _lib.check(lib.px_msa_average(wp.data_ptr(), vp.data_ptr(), got.data_ptr(), s, n, ld, st), "px_msa_average")
    ops.device_error_flags()
    want = torch.softmax(logits.double(), -1) @ v.double()
    relf = lambda a: float((a.double() - want).norm() / want.norm())
    assert (wp[..., n:] == 0).all()
    assert relf(got) < 2 * relf(torch.softmax(logits, -1) @ v) + 1e-7


@pytest.mark.parametrize("s,n", [(1, 1), (5, 17), (40, 33)])
def test_embedding(s, n):
    """px_msa_embed against the linear layer over the concatenated features, for a permuted part of the sequences."""
    torch.manual_seed(s)
    msa = torch.randint(0, 32, (s, n), device="cuda")
    hd, dv = (torch.rand(s, n, device="cuda") for _ in range(2))
    w, sp = torch.randn(64, 34, device="cuda"), torch.randn(n, 64, device="cuda")
    idx = torch.randperm(s, device="cuda")[:max(1, s // 2)]
    x = torch.cat([F.one_hot(msa, 32).double(), hd[..., None].double(), dv[..., None].double()], -1)[idx]
    torch.testing.assert_close(ops.msa_embed(msa, hd, dv, idx, w, sp).double(), x @ w.double().t() + sp.double(), rtol=1e-6, atol=2e-6)
