"""Where modules find their parameters: registered, or as plain attributes and properties (parametrised, flattened, replicated modules)."""
import copy
import gc
import pickle
import weakref

import pytest
import torch
from torch.nn.utils import parametrize

import protenix_b200 as px
from protenix_b200.init_utils import randomize_parameters_


class Twice(torch.nn.Module):
    def forward(self, w):
        return 2 * w


PLACES = ["tri_mul_out.layer_norm_in", "tri_mul_in.linear_a_p", "tri_att_start.mha.linear_q", "tri_att_end.layer_norm", "pair_transition.linear_no_bias",
          "attention_pair_bias.layernorm_z", "attention_pair_bias.attention.linear_k", "single_transition.layernorm1"]


def _flatten(module):
    """The weight as a plain attribute, as wrappers that keep parameters in one flat buffer leave it."""
    w = module._parameters.pop("weight")
    module.weight = w.detach()


def test_layer_norm_finds_parameters_that_are_not_registered():
    """On the CPU the op is refused for that reason and no other."""
    for change in (lambda m: parametrize.register_parametrization(m, "weight", Twice()), _flatten):
        ln = px.LayerNorm(8)
        change(ln)
        with pytest.raises(RuntimeError, match="CUDA"):
            ln(torch.randn(3, 8))


def test_layer_norm_saved_whole_without_its_width_loads():
    """The attribute is younger than saved modules are."""
    ln = px.LayerNorm(8)
    del ln.__dict__["_width"]
    for twin in (copy.deepcopy(ln), pickle.loads(pickle.dumps(ln))):
        with pytest.raises(RuntimeError, match="CUDA"):           # the CPU is refused, and nothing before that fails
            twin(torch.randn(3, 8))


@pytest.mark.gpu
def test_layer_norm_with_a_parametrised_and_a_flattened_weight():
    x, dy = torch.randn(33, 128, device="cuda"), torch.randn(33, 128, device="cuda")
    plain = randomize_parameters_(px.LayerNorm(128), 1).cuda()
    want = plain(x)
    flat = copy.deepcopy(plain)
    _flatten(flat)
    assert torch.equal(flat(x), want)
    double = copy.deepcopy(plain)
    with torch.no_grad():
        double.weight.mul_(2)
    want = torch.autograd.grad(double(x), [double.weight, double.bias], dy)
    parametrize.register_parametrization(plain, "weight", Twice())
    got = torch.autograd.grad(plain(x), [plain.parametrizations.weight.original, plain.bias], dy)
    assert torch.equal(got[0], 2 * want[0]) and torch.equal(got[1], want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("warm", [False, True])
def test_block_with_parametrised_and_flattened_weights(warm):
    n = 40
    s, z = torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda")
    plain, want, flat = (randomize_parameters_(px.PairformerBlock(), 3).cuda().eval() for _ in range(3))
    first = want(s, z, None)
    if warm:                                                      # the change comes after the parameters have been looked up
        plain(s, z, None), flat(s, z, None)
    for place in PLACES:
        parametrize.register_parametrization(plain.get_submodule(place), "weight", Twice())
        _flatten(flat.get_submodule(place))
        with torch.no_grad():
            want.get_submodule(place).weight.mul_(2)
    assert all(torch.equal(a, b) for a, b in zip(flat(s, z, None), first))
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(plain(s, z, None), want(s, z, None)))
    with torch.no_grad():                                         # and the computed weights follow
        plain.get_submodule(PLACES[2]).parametrizations.weight.original.mul_(0.5)
        want.get_submodule(PLACES[2]).weight.mul_(0.5)
    assert all(torch.equal(a, b) for a, b in zip(plain(s, z, None), want(s, z, None)))
    del flat.get_submodule(PLACES[0]).weight
    with pytest.raises(AttributeError):
        flat(s, z, None)


@pytest.mark.gpu
def test_replicas_and_shallow_copies_look_up_their_own_parameters():
    n = 40
    z = torch.randn(n, n, 128, device="cuda")
    for kind in (lambda: px.TriangleAttention(c_in=128, c_hidden=32, no_heads=4), lambda: px.PairformerBlock(c_s=0)):
        call = lambda m: m(z) if isinstance(m, px.TriangleAttention) else m(None, z, None)[1]
        mod, other = (randomize_parameters_(kind(), seed).cuda().eval() for seed in (3, 4))
        want, new = call(mod), call(other)
        with torch.no_grad():
            replica = torch.nn.parallel.replicate(mod, [0])[0]
            twin = copy.copy(mod)
            twin._modules = dict(other._modules)
            mod.load_state_dict({k: v.clone() for k, v in other.state_dict().items()}, assign=True)
        assert torch.equal(call(replica), want)
        assert torch.equal(call(twin), new) and torch.equal(call(mod), new)


def test_kept_look_ups_do_not_keep_their_module_alive():
    """What a module keeps refers to the module's own attributes; with the last reference to the module its parameters are gone."""
    from protenix_b200 import native
    from protenix_b200.msa import MSABlock

    for make, names in ((lambda: px.TriangleAttention(c_in=128, c_hidden=32, no_heads=4), [""]),
                        (lambda: px.OuterProductMean(c_m=64, c_z=128, c_hidden=32), [""]),
                        (lambda: MSABlock(), ["outer_product_mean_msa", "pair_stack.tri_att_end"])):
        mod = make()
        for name in names:
            m = mod.get_submodule(name)
            native.kept(m, lambda: native.params(m, *m.NATIVE))
        if isinstance(mod, MSABlock):
            mod.pair_stack._native()
        held = [weakref.ref(p) for p in mod.parameters()]
        del mod, m
        gc.collect()
        assert not any(r() is not None for r in held)


def test_wrapper_copies_follow_announced_writes_and_new_storages():
    from protenix_b200 import weights

    lin = px.OpenfoldLinear(8, 4, bias=False)
    kept = weights.f16_of(lin.weight)
    lin.weight.data.copy_(torch.ones(4, 8))                       # past the version counter
    px.weights_changed(lin)
    assert weights.f16_of(lin.weight) is not kept and bool((weights.f16_of(lin.weight) == 1).all())
    memory = torch.zeros(64)                                      # two storages over the same memory, one after the other
    over = lambda: torch.from_numpy(memory.numpy())[:32].view(4, 8)
    lin.weight.data = over()
    first, version = weights.f16_of(lin.weight), lin.weight._version
    lin.weight.data = torch.empty(4, 8)
    memory.fill_(3.0)
    lin.weight.data = over()
    assert lin.weight._version == version and lin.weight.data_ptr() == memory.data_ptr()
    assert bool((weights.f16_of(lin.weight) == 3).all()) and bool((first == 0).all())


@pytest.mark.gpu
def test_modules_follow_announced_writes_and_new_storages():
    n = 40
    s, z = torch.randn(n, 384, device="cuda"), torch.randn(n, n, 128, device="cuda")
    blk, other = (randomize_parameters_(px.PairformerBlock(), seed).cuda().eval() for seed in (3, 4))
    first, want = blk(s, z, None), other(s, z, None)
    new = other.state_dict()
    for name, p in blk.named_parameters():                        # an average written over the weights, past the version counters
        p.data.copy_(new[name])
    assert all(torch.equal(a, b) for a, b in zip(blk(s, z, None), first))       # one set or the other, not a mixture
    px.weights_changed(blk.tri_att_start)                         # announced for a part, kept by the block
    px.weights_changed(blk)
    assert all(torch.equal(a, b) for a, b in zip(blk(s, z, None), want))
    old = {k: p.data.clone() for k, p in blk.named_parameters()}
    for name, p in blk.named_parameters():                        # memory given back and taken again, most of it at the same addresses
        p.data = torch.empty(0, device="cuda")
        p.data = torch.empty_like(old[name]).normal_(0, 0.05)
        new[name] = p.data.clone()
    other.load_state_dict(new)
    assert all(torch.equal(a, b) for a, b in zip(blk(s, z, None), other(s, z, None)))


def test_wrappers_tell_devices_apart():
    from protenix_b200 import ops

    here, there = torch.empty(4), torch.empty(4, device="meta")
    ops._one_device(here, None, here)
    with pytest.raises(RuntimeError, match="same device"):
        ops._one_device(here, None, there)


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_inputs_of_another_gpu_than_the_weights_are_refused():
    """On the host, before a launch: also after a call on the right GPU."""
    z, s, far = torch.randn(40, 40, 128), torch.randn(40, 384), "cuda:1"
    blk, ln = px.PairformerBlock().cuda().eval(), px.LayerNorm(128).cuda()
    trunk = px.RecyclingTrunk(n_blocks=0).cuda().eval()
    blk(s.cuda(), z.cuda(), None), ln(z.cuda()), trunk(s.cuda(), z.cuda())
    for call in (lambda: blk(s.to(far), z.to(far), None), lambda: blk(s.to(far), z.cuda(), None), lambda: ln(z.to(far)),
                 lambda: trunk(s.to(far), z.to(far)), lambda: px.dropout_add_rowwise(z.cuda(), z.to(far), 0.5, True)):
        with pytest.raises(RuntimeError, match="same device|device of the other"):
            call()
