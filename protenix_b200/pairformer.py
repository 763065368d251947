"""``PairformerBlock`` / ``PairformerStack`` drop-ins over the sm_100a kernels.

Constructor arguments, forward signature, return values and ``state_dict`` keys are those of
protenix/model/modules/pairformer.py:42-340.  A block is eight kernel families on the pair
tensor (triangle multiplication out/in: projection, contraction, output stage; triangle
attention start/end: projection, flash attention, output stage; transition) plus the small
single-representation branch, issued by the native host path.  z is updated in place on a private
tensor (or on the caller's with ``inplace_safe=True``); the two transposed copies of z the reference makes around
the ending-node attention do not exist here -- the ending-node kernels index z transposed.

Inference only: dropout is the identity (eval mode), gradients are not produced.
"""
from __future__ import annotations

import os
from typing import Optional, Tuple

import torch
import torch.nn as nn

from . import native, ops
from .primitives import Transition
from .transformer import AttentionPairBias
from .triangular import TriangleAttention, TriangleMultiplicationIncoming, TriangleMultiplicationOutgoing


class PairformerBlock(nn.Module):
    def __init__(self, n_heads: int = 16, c_z: int = 128, c_s: int = 384, c_hidden_mul: int = 128,
                 c_hidden_pair_att: int = 32, no_heads_pair: int = 4, num_intermediate_factor: int = 4,
                 dropout: float = 0.25, hidden_scale_up: bool = False) -> None:
        super().__init__()
        self.n_heads = n_heads
        if hidden_scale_up:
            no_heads_pair = c_z // c_hidden_pair_att
            c_hidden_mul = c_z
        self.tri_mul_out = TriangleMultiplicationOutgoing(c_z=c_z, c_hidden=c_hidden_mul)
        self.tri_mul_in = TriangleMultiplicationIncoming(c_z=c_z, c_hidden=c_hidden_mul)
        self.tri_att_start = TriangleAttention(c_in=c_z, c_hidden=c_hidden_pair_att, no_heads=no_heads_pair)
        self.tri_att_end = TriangleAttention(c_in=c_z, c_hidden=c_hidden_pair_att, no_heads=no_heads_pair)
        self.p_drop = dropout
        self.pair_transition = Transition(c_in=c_z, n=num_intermediate_factor)
        self.c_s = c_s
        if self.c_s > 0:
            self.attention_pair_bias = AttentionPairBias(has_s=False, create_offset_ln_z=True, n_heads=n_heads,
                                                         c_a=c_s, c_z=c_z)
            self.single_transition = Transition(c_in=c_s, n=4)

    # the single-representation branch: vectors, then the eight matrices in the order of px_single_prepare
    _V, _A, _T = (ops.C_S,), "attention_pair_bias", "single_transition"
    NATIVE_SINGLE = ("single", [(f"{_A}.layernorm_a.weight", "f", _V), (f"{_A}.layernorm_a.bias", "f", _V),
                      (f"{_A}.attention.linear_q.bias", "f", _V), (f"{_T}.layernorm1.weight", "f", _V),
                      (f"{_T}.layernorm1.bias", "f", _V)]
                     + [(f"attention_pair_bias.attention.linear_{x}.weight", "s", (ops.C_S, ops.C_S)) for x in "qkvgo"]
                     + [(f"single_transition.linear_no_bias_{x}.weight", "s", (4 * ops.C_S, ops.C_S)) for x in "ab"]
                     + [(f"{_T}.linear_no_bias.weight", "s", (ops.C_S, 4 * ops.C_S))],
                     [f"{_A}.layernorm_a.eps", f"{_T}.layernorm1.eps"])

    def _native(self):
        """The native view of this block's parameters."""
        return native.kept(self, self._make_native)

    def _make_native(self):
        for m in (self.tri_mul_out, self.tri_mul_in, self.tri_att_start, self.tri_att_end):
            m._check_shape()
        if (self.pair_transition.c_in, self.pair_transition.n) != (ops.C_Z, 4):
            raise RuntimeError(f"the pair transition kernel is specialised for c_z = {ops.C_Z}, factor 4")
        parts = [native.params(self, *native.under(name, *getattr(self, name).NATIVE))
                 for name in ("tri_mul_out", "tri_mul_in", "tri_att_start", "tri_att_end", "pair_transition")]
        if self._single_kernel():
            parts += [native.params(self, *native.under("attention_pair_bias", *self.attention_pair_bias.NATIVE)),
                      native.params(self, *self.NATIVE_SINGLE)]
        else:
            parts += [None, None]
        return native.load().Block(parts)

    def _single_kernel(self) -> bool:
        """Whether the single branch has the dimensions its kernels are built for."""
        return self.c_s == ops.C_S and self.n_heads == ops.N_HEAD_SINGLE

    def single_path(self, s: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
        """The single-representation update, given the pair bias of the block's final z (it needs nothing else from z), as a
        composition: for other widths and batches than the kernels take."""
        s = s + self.attention_pair_bias(a=s, s=None, z=None, bias=bias)
        return s + self.single_transition(s)

    @torch.no_grad()
    def forward(self, s: Optional[torch.Tensor], z: torch.Tensor, pair_mask: Optional[torch.Tensor],
                triangle_multiplicative: str = "torch", triangle_attention: str = "torch",
                inplace_safe: bool = False, chunk_size: Optional[int] = None
                ) -> Tuple[Optional[torch.Tensor], torch.Tensor]:
        return _run_blocks([self], s, z, pair_mask, inplace_safe)


def _run_blocks(blocks, s: Optional[torch.Tensor], z: torch.Tensor, pair_mask: Optional[torch.Tensor], inplace_safe: bool
                ) -> Tuple[Optional[torch.Tensor], torch.Tensor]:
    for block in blocks:
        if block.training and block.p_drop > 0:
            raise RuntimeError("PairformerBlock: training-mode dropout is not implemented; call .eval()")
    run = native.load().stack_forward
    if s is None or all(b.c_s == 0 or (b._single_kernel() and s.numel() == s.shape[-2] * b.c_s) for b in blocks):
        return run([b._native() for b in blocks], s, z, pair_mask, inplace_safe)
    for block in blocks:
        _, z = run([block._native()], None, z, pair_mask, inplace_safe)
        if block.c_s > 0:
            s = block.single_path(s, block.attention_pair_bias.pair_bias(z))
        inplace_safe = True             # every later block works on the copy the first one made
    return s, z


class PairformerStack(nn.Module):
    def __init__(self, n_blocks: int = 48, n_heads: int = 16, c_z: int = 128, c_s: int = 384,
                 num_intermediate_factor: int = 4, dropout: float = 0.25, blocks_per_ckpt: Optional[int] = None,
                 hidden_scale_up: bool = False) -> None:
        super().__init__()
        self.n_blocks = n_blocks
        self.n_heads = n_heads
        self.blocks_per_ckpt = blocks_per_ckpt
        self.blocks = nn.ModuleList(
            PairformerBlock(n_heads=n_heads, c_z=c_z, c_s=c_s, num_intermediate_factor=num_intermediate_factor,
                            dropout=dropout, hidden_scale_up=hidden_scale_up) for _ in range(n_blocks))

    @torch.no_grad()
    def forward(self, s: torch.Tensor, z: torch.Tensor, pair_mask: Optional[torch.Tensor],
                triangle_multiplicative: str = "torch", triangle_attention: str = "torch",
                inplace_safe: bool = False, chunk_size: Optional[int] = None
                ) -> Tuple[torch.Tensor, torch.Tensor]:
        s, z = _run_blocks(list(self.blocks), s, z, pair_mask, inplace_safe)
        if os.environ.get("PX_CHECK_DEVICE_ERRORS", "0") == "1":    # synchronises: off unless asked for
            ops.device_error_flags(z.device)
        return s, z
