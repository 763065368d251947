"""The single-representation branch (px_single_update) against the torch composition of the same modules in fp64, and no
further from it than the composition in fp32."""
import pytest
import torch

import protenix_b200 as px
from protenix_b200 import ops
from protenix_b200.init_utils import randomize_parameters_

pytestmark = pytest.mark.gpu


def _composition(blk, s, bias, dt):
    from torch.nn import functional as F

    att, tr = blk.attention_pair_bias, blk.single_transition
    a, g = att.attention, (lambda p: p.detach().to(dt))
    s, bias, n = s.to(dt), bias.to(dt), s.shape[0]
    heads = lambda w, b=None: F.linear(x, g(w.weight), b).view(n, 16, 24).transpose(0, 1)
    x = F.layer_norm(s, (384,), g(att.layernorm_a.weight), g(att.layernorm_a.bias), att.layernorm_a.eps)
    q, k, v = heads(a.linear_q, g(a.linear_q.bias)), heads(a.linear_k), heads(a.linear_v)
    o = torch.softmax(q / 24 ** 0.5 @ k.transpose(-1, -2) + bias, -1) @ v
    o = o.transpose(0, 1).reshape(n, 384) * torch.sigmoid(F.linear(x, g(a.linear_g.weight)))
    s = s + F.linear(o, g(a.linear_o.weight))
    y = F.layer_norm(s, (384,), g(tr.layernorm1.weight), g(tr.layernorm1.bias), tr.layernorm1.eps)
    h = F.silu(F.linear(y, g(tr.linear_no_bias_a.weight))) * F.linear(y, g(tr.linear_no_bias_b.weight))
    return s + F.linear(h, g(tr.linear_no_bias.weight))


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 64, 65, 127, 128, 129, 200, 390])
def test_single_update(n):
    torch.manual_seed(n)
    blk = randomize_parameters_(px.PairformerBlock(), 3).cuda().eval()
    s, bias = torch.randn(n, 384, device="cuda"), 3 * torch.randn(16, n, n, device="cuda")
    relf = lambda a, b: float((a.double() - b).norm() / b.norm())
    with torch.no_grad():
        want = _composition(blk, s, bias, torch.float64)
        got = blk.single_path(s, bias)
        ops.device_error_flags()
        assert relf(got, want) < 2 * relf(_composition(blk, s, bias, torch.float32), want) + 1e-7
        assert torch.equal(got, blk.single_path(s, bias))
        for dt in (torch.bfloat16, torch.float16):
            sd = s.to(dt)
            out = blk.single_path(sd[None], bias)
            assert out.dtype == dt and out.shape == (1, n, 384)
            assert relf(out[0], _composition(blk, sd, bias, torch.float64)) < 6e-3
