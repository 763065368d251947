"""The ways in which the output stages' rows leave give the same bits: added in place, stored without a residual, and with the residual of
another tensor.  The triangle kernels write fp32 rows of the last kind with plain accesses, everything else leaves by TMA (the transition
has its residual fetched by TMA into the staging area).  The modules' in-place forms and the tensor wrappers agree as well."""
import pytest
import torch

import protenix_b200 as px
from protenix_b200 import ops
from protenix_b200.init_utils import randomize_parameters_

pytestmark = pytest.mark.gpu


def _modules():
    return [randomize_parameters_(m, 5).cuda().eval() for m in (
        px.TriangleMultiplicationOutgoing(c_z=128, c_hidden=128), px.TriangleAttention(c_in=128, c_hidden=32, no_heads=4),
        px.TriangleAttention(c_in=128, c_hidden=32, no_heads=4, starting=False), px.Transition(c_in=128, n=4))]


@pytest.mark.parametrize("n", [1, 31, 33, 129, 160, 257])
def test_stored_added_and_plain_rows_agree(n):
    torch.manual_seed(n)
    z = torch.randn(n, n, 128, device="cuda")
    mask = torch.ones(n, n, device="cuda")
    mul, start, end, tr = _modules()
    with torch.no_grad():
        for name in ("mul", "start", "end", "transition"):
            if name == "mul":
                run = lambda a, b, add: ops.triangle_multiplication(a, b, mask, *mul._kernel_args(), incoming=False, add_residual=add)
            elif name == "transition":
                run = lambda a, b, add: ops.transition(a, b, *tr._weights(), add_residual=add)
            else:
                mod = start if name == "start" else end
                run = lambda a, b, add: ops.triangle_attention(a, b, mask, *mod._kernel_args(), ending=name == "end", add_residual=add)
            plain, update, added = torch.empty_like(z), torch.full_like(z, float("nan")), z.clone()
            run(z, plain, True)
            run(z, update, False)
            run(added, added, True)
            ops.device_error_flags()
            assert torch.equal(added, plain), name
            assert torch.equal(z + update, plain), name
            zm = z.clone()
            same = (mul.apply_(zm, mask) if name == "mul" else tr.forward_residual_(zm) if name == "transition" else
                    mod.apply_(zm, mask, ending=name == "end"))
            assert same.data_ptr() == zm.data_ptr() and torch.equal(zm, plain), name


@pytest.mark.parametrize("rows", [1, 31, 128, 129, 1000])
def test_bf16_transition_without_residual(rows):
    """bf16 rows: the update alone is the fp32 one rounded, and a residual is added before the rounding."""
    torch.manual_seed(rows)
    x = torch.randn(rows, 128, device="cuda").bfloat16()
    tr = randomize_parameters_(px.Transition(c_in=128, n=4), 5).cuda().eval()
    update, zero, fp32 = torch.full_like(x, float("nan")), torch.empty_like(x), torch.empty(rows, 128, device="cuda")
    with torch.no_grad():
        ops.transition(x, update, *tr._weights(), add_residual=False)
        ops.transition(x, zero, *tr._weights(), add_residual=True)
        ops.transition(x.float(), fp32, *tr._weights(), add_residual=False)
    ops.device_error_flags()
    assert torch.equal(update, fp32.bfloat16())
    assert torch.equal(zero, (x.float() + fp32).bfloat16())
