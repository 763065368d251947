"""Performance cases of the package: the calls its users make, at the sizes they make them.

Structure prediction runs the trunk on complexes of some dozens to some 1500 tokens, with the pair tensor z stored in
fp32 (the default) or bf16; complexes have any length and come padded.  The trunk is 48 Pairformer blocks per recycling
cycle with the MSA module in front; the confidence head is a stack of 4 blocks.  The triangle modules, the transition,
the LayerNorm op and the dropout-add are also used alone, as drop-ins inside other models and in training code.

A model is built once per configuration and kept for all inputs, as a serving or training process keeps it; its weights
are re-drawn because freshly initialised blocks are the identity.  Inputs differ by seed.
"""
from __future__ import annotations

import math

import torch

import protenix_b200 as px
from protenix_b200.fused_ops import dropout_add_rowwise
from protenix_b200.init_utils import randomize_parameters_
from protenix_b200.msa import MSAModule

C_Z, C_S, C_S_INPUTS, C_M = 128, 384, 449, 64
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
SIZE = {"fp32": 4, "bf16": 2}
P_DROP = 0.25


def listed():
    return [
        # The single representation's LayerNorm: the smallest call of the package, nothing but latency.
        {"name": "layer_norm_single", "op": "layer_norm", "rows": 384, "cols": C_S, "dtype": "fp32", "train": False},
        # LayerNorm over a pair tensor in a training step: forward with statistics, then dx, dgamma, dbeta.
        {"name": "layer_norm_train", "op": "layer_norm", "rows": 768 * 768, "cols": C_Z, "dtype": "bf16", "train": True},
        # Residual + row-shared dropout of a training step (crop of 512 tokens), forward and backward.
        {"name": "dropout_add_train", "op": "dropout_add", "n": 512, "dtype": "bf16"},
        # The pair transition alone, as a module returns it (no residual).
        {"name": "transition_1024", "op": "transition", "n": 1024, "dtype": "bf16"},
        # Outgoing, then incoming triangle multiplication at N=768 with the last tenth of the tokens padded.
        {"name": "tri_mul_768", "op": "tri_mul", "n": 768, "pad": 77, "dtype": "bf16"},
        # Starting-node, then ending-node triangle attention, same inputs.
        {"name": "tri_att_768", "op": "tri_att", "n": 768, "pad": 77, "dtype": "bf16"},
        # One block on a small protein: launches and host time count.
        {"name": "block_128", "op": "stack", "n": 128, "pad": 0, "blocks": 1, "dtype": "fp32"},
        # One block on an odd length with odd padding, pair tensor in bf16.
        {"name": "block_437_ragged", "op": "stack", "n": 437, "pad": 19, "blocks": 1, "dtype": "bf16"},
        # The full stack on an ordinary protein.
        {"name": "stack48_384", "op": "stack", "n": 384, "pad": 0, "blocks": 48, "dtype": "fp32"},
        # The confidence head's depth on the largest complex of the benchmark, 37 padded tokens.
        {"name": "stack4_1536", "op": "stack", "n": 1536, "pad": 37, "blocks": 4, "dtype": "fp32"},
        # The MSA module: 4 blocks, 1024 sequences.
        {"name": "msa_384x1024", "op": "msa", "n": 384, "n_msa": 1024, "dtype": "fp32"},
        # The whole trunk with recycling on a short chain: 4 cycles of MSA module and 48 blocks.
        {"name": "trunk_200x512", "op": "trunk", "n": 200, "n_msa": 512, "cycles": 4, "dtype": "fp32"},
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _pad(rng, n):
    """Padding as it comes: none, a few tokens, or up to a tenth."""
    return rng.choice([0, rng.randint(0, min(64, n // 8)), rng.randint(0, n // 10)])


def draw(rng):
    op = rng.choice(["layer_norm", "layer_norm", "dropout_add", "transition", "tri_mul", "tri_att", "stack", "stack",
                     "stack", "stack", "msa", "trunk"])
    dtype = rng.choice(["fp32", "bf16"])
    if op == "layer_norm":
        return {"op": op, "rows": _log(rng, 64, 768 * 768), "cols": rng.choice([C_M, C_Z, C_S]), "dtype": dtype,
                "train": rng.random() < 0.5}
    if op == "dropout_add":
        return {"op": op, "n": _log(rng, 64, 768), "dtype": dtype}
    if op == "transition":
        return {"op": op, "n": _log(rng, 24, 1536), "dtype": dtype}
    if op in ("tri_mul", "tri_att"):
        n = _log(rng, 24, 1536)
        return {"op": op, "n": n, "pad": _pad(rng, n), "dtype": dtype}
    if op == "stack":
        blocks = rng.choice([1, 4, 48])
        n = _log(rng, 24, {1: 1536, 4: 1400, 48: 512}[blocks])
        return {"op": op, "n": n, "pad": _pad(rng, n), "blocks": blocks, "dtype": "fp32" if blocks > 4 else dtype}
    n = _log(rng, 24, 600 if op == "msa" else 224)
    case = {"op": op, "n": n, "n_msa": _log(rng, 32, 2048 if op == "msa" else 1024), "dtype": "fp32"}
    if op == "trunk":
        case["cycles"] = rng.randint(1, 4)
    return case


_MODELS = {}


def _model(key, make):
    """The model of one configuration, built on first use and kept (this module's stand-in for a user's process)."""
    if key not in _MODELS:
        _MODELS[key] = make()
    return _MODELS[key]


def _ready(module):
    return randomize_parameters_(module, 1).cuda().eval()


# all rows in their order, however many there are: a pass draws nothing
MSA_CONFIGS = {"strategy": "topk", "min_size": {"train": 1 << 20, "test": 1 << 20}}


def _msa_inputs(n, n_msa, gen):
    msa = torch.randint(0, 31, (n_msa, n), generator=gen, device="cuda")
    msa[torch.rand(n_msa, n, generator=gen, device="cuda") < 0.2] = 31          # gaps
    deletion = (torch.rand(n_msa, n, generator=gen, device="cuda") < 0.05).float()
    return {"msa": msa, "has_deletion": deletion,
            "deletion_value": deletion * torch.rand(n_msa, n, generator=gen, device="cuda")}


def _mask(n, pad):
    valid = torch.ones(n, device="cuda")
    valid[n - pad:] = 0
    return valid[:, None] * valid[None, :]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    op, dt = case["op"], DTYPES[case["dtype"]]
    state = {"op": op}
    if op == "layer_norm":
        cols, train = case["cols"], case["train"]
        state["model"] = _model((op, cols), lambda: _ready(px.LayerNorm(cols)))
        # activations: not centred, rows of unlike scale
        state["x"] = ((0.5 + normal(case["rows"], cols)) * (0.5 + normal(case["rows"], 1).abs())).to(dt)
        state["x"].requires_grad_(train)
        state["train"] = train
        if train:
            state["dy"] = normal(case["rows"], cols).to(dt)
        return state
    n = case["n"]
    z = normal(n, n, C_Z).to(dt)
    if op == "dropout_add":
        state.update(residual=z.requires_grad_(), x=normal(n, n, C_Z).to(dt).requires_grad_(),
                     grad=normal(n, n, C_Z).to(dt), seed=seed)
        return state
    state["z"] = z
    if op == "transition":
        state["model"] = _model(op, lambda: _ready(px.Transition(c_in=C_Z, n=4)))
        return state
    if op == "tri_mul":
        state["model"] = _model(op, lambda: [_ready(px.TriangleMultiplicationOutgoing(c_z=C_Z, c_hidden=C_Z)),
                                             _ready(px.TriangleMultiplicationIncoming(c_z=C_Z, c_hidden=C_Z))])
        state["mask"] = _mask(n, case["pad"])
        return state
    if op == "tri_att":
        state["model"] = _model(op, lambda: [_ready(px.TriangleAttention(c_in=C_Z, c_hidden=32, no_heads=4, starting=s))
                                             for s in (True, False)])
        state["mask"] = _mask(n, case["pad"])
        return state
    if op == "stack":
        blocks = case["blocks"]
        state["model"] = _model((op, blocks), lambda: _ready(px.PairformerBlock() if blocks == 1
                                                             else px.PairformerStack(n_blocks=blocks)))
        state.update(s=normal(n, C_S), mask=_mask(n, case["pad"]))
        return state
    n_msa = case["n_msa"]
    state.update(features=_msa_inputs(n, n_msa, gen), s_inputs=normal(n, C_S_INPUTS), mask=_mask(n, 0))
    if op == "msa":
        state["model"] = _model(op, lambda: _ready(MSAModule(n_blocks=4, c_s_inputs=C_S_INPUTS,
                                                             msa_configs=MSA_CONFIGS)))
    else:
        state["model"] = _model(op, lambda: _ready(px.RecyclingTrunk(n_blocks=48, msa_n_blocks=4,
                                                                     c_s_inputs=C_S_INPUTS, msa_configs=MSA_CONFIGS)))
        state.update(s=normal(n, C_S), cycles=case["cycles"])
    return state


def run(state):
    op = state["op"]
    if op == "layer_norm" and state["train"]:
        model, x = state["model"], state["x"]
        y = model(x)
        return (y,) + torch.autograd.grad(y, [x, model.weight, model.bias], state["dy"])
    if op == "dropout_add":
        torch.cuda.manual_seed(state["seed"])
        out = dropout_add_rowwise(state["residual"], state["x"], P_DROP, True)
        return (out,) + torch.autograd.grad(out, [state["residual"], state["x"]], state["grad"])
    model = state["model"]
    with torch.no_grad():
        if op == "layer_norm":
            return model(state["x"])
        if op == "transition":
            return model(state["z"])
        if op in ("tri_mul", "tri_att"):
            return [m(state["z"], state["mask"]) for m in model]
        if op == "stack":
            return model(state["s"], state["z"], state["mask"])
        if op == "msa":
            return model(state["features"], state["z"], state["s_inputs"], state["mask"])
        return model(state["s"], state["z"], state["mask"], N_cycle=state["cycles"],
                     input_feature_dict=state["features"], s_inputs=state["s_inputs"])


# ------------------------------------------------------------------------------------------------------------------
# Work of one pass: inputs, weights and outputs once each; multiplications and additions of the matrix products.
def _pair_block_flops(n):
    return 1536 * n ** 3 + 1121792 * n ** 2


def _single_flops(n):
    return n * (5 * 2 * C_S * C_S + 3 * 2 * C_S * 4 * C_S) + 4 * n * n * C_S + 2 * 16 * C_Z * n * n


def _msa_flops(n, s):
    """4 blocks: outer product mean, pair-weighted averaging and transition of the MSA (not in the last), pair block."""
    outer = 2 * 1024 * s * n * n + 2 * 1024 * C_Z * n * n
    msa = 2 * C_M * s * n * n + s * n * (2 * 3 * C_M * C_M + 3 * 2 * C_M * 4 * C_M)
    return 4 * (outer + _pair_block_flops(n)) + 3 * msa


PAIR_BLOCK_WEIGHTS = 2 * 6 * C_Z * C_Z + 2 * 5 * C_Z * C_Z + 12 * C_Z * C_Z
SINGLE_WEIGHTS = 5 * C_S * C_S + 12 * C_S * C_S


def work(case):
    op = case["op"]
    e = SIZE[case["dtype"]]
    if op == "layer_norm":
        t = case["rows"] * case["cols"]
        # forward: x, y; backward: dy, x, dx
        return {"bytes": t * e * (5 if case["train"] else 2), "flops": t * (20 if case["train"] else 8)}
    n = case["n"]
    z = n * n * C_Z * e
    if op == "dropout_add":
        return {"bytes": 5 * z, "flops": 3 * n * n * C_Z}      # residual, x, out; gradient, dx
    if op == "transition":
        return {"bytes": 2 * z + 4 * 12 * C_Z * C_Z, "flops": 393216 * n * n}
    mask = 4 * n * n
    if op == "tri_mul":
        return {"bytes": 2 * (2 * z + mask + 4 * 6 * C_Z * C_Z), "flops": 2 * (256 * n ** 3 + 196608 * n * n)}
    if op == "tri_att":
        return {"bytes": 2 * (2 * z + mask + 4 * 5 * C_Z * C_Z), "flops": 2 * (512 * n ** 3 + 164864 * n * n)}
    if op == "stack":
        b = case["blocks"]
        return {"bytes": 2 * z + mask + 8 * n * C_S + b * 4 * (PAIR_BLOCK_WEIGHTS + SINGLE_WEIGHTS),
                "flops": b * (_pair_block_flops(n) + _single_flops(n))}
    s = case["n_msa"]
    inputs = 16 * n * s + mask + 4 * n * C_S_INPUTS
    msa_weights = 4 * 4 * (PAIR_BLOCK_WEIGHTS + 1024 * C_Z + 16 * C_M * C_M)
    if op == "msa":
        return {"bytes": 2 * z + inputs + msa_weights, "flops": _msa_flops(n, s)}
    c = case["cycles"]
    return {"bytes": 2 * z + inputs + 8 * n * C_S + msa_weights + 48 * 4 * (PAIR_BLOCK_WEIGHTS + SINGLE_WEIGHTS),
            "flops": c * (_msa_flops(n, s) + 48 * (_pair_block_flops(n) + _single_flops(n)) + 2 * C_Z * C_Z * n * n)}


def tolerance(case):
    """The matrix products take 16-bit operands with fp32 sums: against an fp64 oracle a block on an fp32 pair tensor is
    off by 6e-4 and 48 blocks by 4e-3 (errors of independent blocks add in squares), on a bf16 one a block by 5.5e-3."""
    op, bf16 = case["op"], case["dtype"] == "bf16"
    if op == "layer_norm":
        # dgamma and dbeta are sums over all rows
        return {"rel": 5e-3 if bf16 else 3e-5 if case["train"] else 1e-5, "max": 0.05 if bf16 else 1e-3}
    if op == "dropout_add":
        return {"rel": 5e-3 if bf16 else 1e-6}
    if op in ("transition", "tri_mul", "tri_att"):
        return {"rel": 1e-2 if bf16 else 2e-3}
    if op == "stack":
        return {"rel": (1e-2 if bf16 else 2e-3) * math.sqrt(min(case["blocks"], 48))}
    return {"rel": 5e-3 if op == "msa" else 2e-2}
