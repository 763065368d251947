"""The single-representation branch (px_single_project, px_single_finish) against the torch composition of the same modules in fp64, and no
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
    s, z = torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda")
    relf = lambda a, b: float((a.double() - b).norm() / b.norm())
    got, z_out = blk(s, z, None)
    ops.device_error_flags()
    with torch.no_grad():
        bias = blk.attention_pair_bias.pair_bias(z_out)          # all the branch takes from z
        want = _composition(blk, s, bias, torch.float64)
        assert relf(got, want) < 2 * relf(_composition(blk, s, bias, torch.float32), want) + 1e-7
        assert torch.equal(got, blk(s, z, None)[0])
        for dt in (torch.bfloat16, torch.float16):
            sd = s.to(dt)
            out = blk(sd[None], z[None], None)[0]
            assert out.dtype == dt and out.shape == (1, n, 384)
            assert relf(out[0], _composition(blk, sd, bias, torch.float64)) < 6e-3


def test_parameters_are_followed():
    """The native view of a module notices new values, storages, parameter objects and submodules; a copy has its own."""
    import copy

    torch.manual_seed(0)
    blk = randomize_parameters_(px.PairformerBlock(), 3).cuda().eval()
    s, z = torch.randn(40, 384, device="cuda"), torch.randn(40, 40, 128, device="cuda")
    other = randomize_parameters_(px.PairformerBlock(), 4).cuda().eval()
    first, want = blk(s, z, None), other(s, z, None)
    assert not torch.equal(first[1], want[1])
    twin = copy.deepcopy(blk)
    assert torch.equal(twin(s, z, None)[1], first[1])
    blk.load_state_dict(other.state_dict())                                      # new values in place
    assert all(torch.equal(a, b) for a, b in zip(blk(s, z, None), want))
    assert torch.equal(twin(s, z, None)[1], first[1])
    twin.load_state_dict(other.state_dict(), assign=True)                        # new parameter objects
    assert all(torch.equal(a, b) for a, b in zip(twin(s, z, None), want))
    third = randomize_parameters_(px.PairformerBlock(), 3).cuda().eval()
    assert torch.equal(third(s, z, None)[1], first[1])
    for name, sub in other.named_children():                                     # new submodules
        setattr(third, name, sub)
    assert all(torch.equal(a, b) for a, b in zip(third(s, z, None), want))
    stack = px.PairformerStack(n_blocks=1).eval()
    stack.blocks[0] = third
    keep = z.clone()
    assert all(torch.equal(a, b) for a, b in zip(stack(s, z, None), want)) and torch.equal(z, keep)
    out = stack(s, z, None, inplace_safe=True)
    assert out[1].data_ptr() == z.data_ptr() and torch.equal(z, want[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 64), (7, 72), (5, 128), (300, 256), (33, 384), (9, 512), (130, 640), (64, 100)])
def test_layer_norm_gradients_with_fp32_parameters(rows, cols, dtype):
    """The backward's register, row-group and wide forms, with fp32 parameters rounded to the type of x."""
    torch.manual_seed(cols)
    ln = randomize_parameters_(px.LayerNorm(cols), 2).cuda()
    x = (2 * torch.randn(rows, cols, device="cuda") + 1).to(dtype).requires_grad_()
    dy = torch.randn(rows, cols, device="cuda").to(dtype)
    y = ln(x)
    got = torch.autograd.grad(y, [x, ln.weight, ln.bias], dy)
    assert got[1].dtype == torch.float32 and got[0].dtype == dtype
    x64 = x.detach().double().requires_grad_()
    w64, b64 = (p.detach().to(dtype).double().requires_grad_() for p in (ln.weight, ln.bias))
    y64 = torch.nn.functional.layer_norm(x64, (cols,), w64, b64, 1e-5)
    want = torch.autograd.grad(y64, [x64, w64, b64], dy.double())
    tol = 2e-6 if dtype == torch.float32 else 6e-3 if dtype == torch.bfloat16 else 1e-3
    for a, b in zip((y,) + got, (y64,) + want):
        assert float((a.double() - b).norm() / b.norm().clamp_min(1e-30)) < tol
