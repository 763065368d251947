"""fp32 rows that leave by TMA (added in place, or without a residual) against the plain accesses (residual in another tensor)."""
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
