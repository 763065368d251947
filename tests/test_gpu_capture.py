"""Capture of module calls into CUDA graphs: replays give what a plain call gives, and nothing that a capture leaves behind is kept for later calls."""
import gc
import time

import pytest
import torch

import protenix_b200 as px
from protenix_b200 import ops, weights
from protenix_b200.init_utils import randomize_parameters_
from protenix_b200.msa import MSAModule

pytestmark = pytest.mark.gpu

N, N_MSA = 40, 24
TOPK = {"strategy": "topk", "min_size": {"train": 1 << 20, "test": 1 << 20}}


def _ready(module, seed=3):
    return randomize_parameters_(module, seed).cuda().eval()


def _features():
    return {"msa": torch.randint(0, 32, (N_MSA, N), device="cuda"), "has_deletion": torch.zeros(N_MSA, N, device="cuda"),
            "deletion_value": torch.rand(N_MSA, N, device="cuda")}


def _case(name, dtype):
    """(module, call of static inputs s and z)"""
    mask = torch.ones(N, N, device="cuda")
    mask[N - 3:] = mask[:, N - 3:] = 0
    if name == "block":
        m = _ready(px.PairformerBlock())
        return m, lambda s, z: m(s, z, mask)
    if name == "stack":
        m = _ready(px.PairformerStack(n_blocks=3))
        return m, lambda s, z: m(s, z, mask)
    if name == "tri_mul":
        m = _ready(px.TriangleMultiplicationIncoming(c_z=128, c_hidden=128))
        return m, lambda s, z: (m(z, mask),)
    if name == "tri_att":
        m = _ready(px.TriangleAttention(c_in=128, c_hidden=32, no_heads=4, starting=False))
        return m, lambda s, z: (m(z, mask),)
    if name == "transition":
        m = _ready(px.Transition(c_in=128, n=4))
        return m, lambda s, z: (m(z),)
    feat, s_inputs = _features(), torch.randn(N, 449, device="cuda")
    if name == "msa":
        m = _ready(MSAModule(n_blocks=2, msa_configs=TOPK))
        return m, lambda s, z: (m(feat, z, s_inputs, mask),)
    m = _ready(px.RecyclingTrunk(n_blocks=2, N_cycle=2, msa_n_blocks=2, msa_configs=TOPK))
    return m, lambda s, z: m(s, z, mask, input_feature_dict=feat, s_inputs=s_inputs)


def _inputs(dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(N, 384, generator=g, device="cuda"), torch.randn(N, N, 128, generator=g, device="cuda").to(dtype)


def _warm_up(call, s, z):
    """As the framework's documentation does it: on a stream that is not the one of the capture."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(s, z)
    torch.cuda.current_stream().wait_stream(side)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", ["block", "stack", "tri_mul", "tri_att", "transition", "msa", "trunk"])
def test_replays_equal_plain_calls(name, dtype):
    torch.manual_seed(1)
    _, call = _case(name, dtype)
    s, z = _inputs(dtype)
    _warm_up(call, s, z)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(s, z)
    for seed in (1, 2):
        new = _inputs(dtype, seed)
        s.copy_(new[0])
        z.copy_(new[1])
        graph.replay()
        got = [t.clone() for t in out]
        want = call(*new)
        ops.device_error_flags()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", ["block", "tri_att", "trunk"])
def test_first_call_under_capture_is_refused(name):
    """Weights laid out inside a capture would be written by replays alone: the call says so, and plain calls are not touched by it."""
    torch.manual_seed(1)
    module, call = _case(name, torch.float32)
    s, z = _inputs(torch.float32)
    with pytest.raises(RuntimeError, match="capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            call(s, z)
    first = call(s, z)
    module.load_state_dict({k: v.clone() for k, v in module.state_dict().items()}, assign=True)
    assert all(torch.equal(a, b) for a, b in zip(first, call(s, z)))
    with torch.no_grad():
        for p in module.parameters():                             # changed since: refused again
            p.mul_(1.0)
    with pytest.raises(RuntimeError, match="capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            call(s, z)
    assert all(torch.equal(a, b) for a, b in zip(first, call(s, z)))


def test_a_graph_keeps_the_weights_it_was_captured_with():
    blk = _ready(px.PairformerBlock())
    s, z = _inputs(torch.float32)
    old = {k: v.clone() for k, v in blk.state_dict().items()}
    want = [t.clone() for t in blk(s, z, None)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = blk(s, z, None)
    blk.load_state_dict(randomize_parameters_(px.PairformerBlock(), 9).state_dict())
    other = blk(s, z, None)                                       # lays out the new weights and lets go of the old ones
    junk = [torch.full((1 << 18,), float("nan"), device="cuda") for _ in range(64)]
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(out, want)) and not torch.equal(other[1], want[1])
    del junk, out, other
    blk.load_state_dict(old)
    assert all(torch.equal(a, b) for a, b in zip(blk(s, z, None), want))
    held = torch.cuda.memory_allocated()
    del graph
    gc.collect()
    for _ in range(100):                                          # the driver lets go of it in a thread of its own
        torch.cuda.synchronize()
        blk(s, z, None)
        if torch.cuda.memory_allocated() < held - (1 << 20):
            return
        time.sleep(0.02)
    raise AssertionError("the weights of a graph's capture outlive the graph")


def test_wrappers_keep_nothing_of_a_capture():
    """The tensor wrappers' 16-bit copies and workspaces: made inside a capture, they are that graph's alone."""
    weights.clear()
    ops.release_workspaces()
    mul = _ready(px.TriangleMultiplicationOutgoing(c_z=128, c_hidden=128))
    _, z = _inputs(torch.float32)
    out = torch.empty_like(z)
    with torch.no_grad():
        run = lambda: ops.triangle_multiplication(z, out, None, *args, incoming=False, add_residual=False)
        args = mul._kernel_args()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        assert not weights._cache and not ops._workspaces
        want = run().clone()
        for _ in range(2):
            out.zero_()
            graph.replay()
            assert torch.equal(out, want)
        ops.release_workspaces()
        weights.clear()
        junk = [torch.full((1 << 18,), float("nan"), device="cuda") for _ in range(64)]
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
        del junk
