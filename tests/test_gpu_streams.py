"""Weights kept between calls, used and renewed on several streams."""
import threading

import pytest
import torch

import protenix_b200 as px
from protenix_b200 import ops, weights
from protenix_b200.init_utils import randomize_parameters_

pytestmark = pytest.mark.gpu

DELAY = 600_000_000          # clock cycles of a waiting kernel: some 0.3 s, against some milliseconds of host work


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_renewed_weights_leave_calls_in_flight_alone(dtype):
    """A call waits on one stream while the weights are changed and laid out anew on another: it still gets the old ones."""
    n = 40
    blk = randomize_parameters_(px.PairformerBlock(), 3).cuda().eval()
    s, z = torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda").to(dtype)
    want = [t.clone() for t in blk(s, z, None)]                   # the weights are laid out on this stream
    new = randomize_parameters_(px.PairformerBlock(), 9).cuda().state_dict()
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
        blk(s, z, None)                                           # so that nothing has to be allocated later
        torch.cuda._sleep(DELAY)
        late = blk(s, z, None)
    blk.load_state_dict(new)
    now = blk(s, z, None)
    waiting = not other.query()
    torch.cuda.synchronize()
    ops.device_error_flags()
    assert all(torch.equal(a, b) for a, b in zip(late, want)) and not torch.equal(now[1], want[1])
    if not waiting:
        pytest.skip("the host took longer than the delay: nothing was in flight")


def test_16_bit_copies_across_streams():
    p = torch.nn.Parameter(torch.randn(128, 128, device="cuda"))
    fill = lambda: [torch.full((128, 128), float("nan"), dtype=torch.float16, device="cuda") for _ in range(64)]
    with torch.no_grad():                                         # loads every kernel used below, which may wait for the device
        p.add_(p.half().clone()).add_(1.0)
    fill()
    torch.cuda.synchronize()
    torch.cuda._sleep(DELAY)
    first = weights.f16_of(p)                                     # converted after the delay
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        assert weights.f16_of(p) is first
        seen = first.clone()
        torch.cuda._sleep(DELAY)
        late = first.clone()
    torch.cuda.current_stream().synchronize()
    want = p.detach().half()
    with torch.no_grad():
        p.add_(1.0)
    del first
    junk = [weights.f16_of(p)] + fill()
    waiting = not other.query()
    torch.cuda.synchronize()
    assert torch.equal(seen, want) and torch.equal(late, want)
    assert torch.equal(junk[0], p.detach().half())
    if not waiting:
        pytest.skip("the host took longer than the delay: nothing was in flight")


def test_threads_share_a_module_while_its_weights_are_renewed():
    """Several threads call one stack on streams of their own; one of them lays the (same) weights out anew again and again."""
    n = 40
    stack = randomize_parameters_(px.PairformerStack(n_blocks=2), 3).cuda().eval()
    inputs = [(torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda")) for _ in range(4)]
    want = [stack(s, z, None) for s, z in inputs]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for k in range(30):
                if i == 0:
                    px.weights_changed(stack)
                got = stack(*inputs[i], None)
                stream.synchronize()
                if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                    wrong.append((i, k))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ops.device_error_flags()
    assert not wrong
