"""The stack runs the single branch of a block beside the attention core of the next one, above 1280 tokens in order; block by block, on one
stream, the same bits."""
import pytest
import torch

import protenix_b200 as px
from protenix_b200 import ops
from protenix_b200.init_utils import randomize_parameters_

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, blocks", [(1, 3), (40, 1), (40, 2), (130, 4), (257, 3), (769, 2), (1281, 2)])
def test_stack_equals_its_blocks(n, blocks, dtype):
    torch.manual_seed(n)
    stack = randomize_parameters_(px.PairformerStack(n_blocks=blocks), 3).cuda().eval()
    s, z = torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda").to(dtype)
    mask = (torch.rand(n, n, device="cuda") < 0.9).float()
    with torch.no_grad():
        want = (s.clone(), z.clone())
        for block in stack.blocks:
            want = block(want[0], want[1], mask)
        for _ in range(3):                                   # the branch meets the pair path elsewhere from call to call
            got = stack(s, z, mask)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    ops.device_error_flags()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, blocks", [(40, 9), (64, 20), (130, 13), (384, 17), (385, 4), (641, 5)])
def test_pair_bias_buffers_are_written_anew_in_time(n, blocks, dtype):
    """Up to 384 tokens eight pair-bias buffers take turns and the main stream waits for the side stream once in four blocks, from the ninth
    block on; beyond there are two, and it waits from the third on.  A buffer written too early changes the update that still reads it."""
    test_stack_equals_its_blocks(n, blocks, dtype)
