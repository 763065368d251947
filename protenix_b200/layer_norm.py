"""LayerNorm modules backed by ``px_layer_norm_fwd_params``.

Same constructor, parameter names and forward as the reference's ``FusedLayerNorm``
(protenix/model/layer_norm/layer_norm.py:199-233) and its ``LayerNorm`` factory
(protenix/model/triangular/layers.py:246-256).  Under ``torch.no_grad()`` (the inference path) the forward is one
kernel launch; when gradients are wanted the op runs as a native autograd function whose backward is
``px_layer_norm_bwd_params`` (the reference's ``FusedLayerNormAffineFunction``, layer_norm.py:69-196).
"""
from __future__ import annotations

import numbers
from typing import Optional, Union

import torch
from torch.nn.parameter import Parameter

from . import native


def _layer_norm(*args):
    """The native op; the first call puts it in this function's place."""
    global _layer_norm
    _layer_norm = native.load().layer_norm
    return _layer_norm(*args)


class FusedLayerNorm(torch.nn.Module):
    def __init__(self, normalized_shape: Union[int, list, torch.Size], create_scale: bool = True,
                 create_offset: bool = True, eps: float = 1e-5) -> None:
        super().__init__()
        if isinstance(normalized_shape, numbers.Integral):
            normalized_shape = (normalized_shape,)
        self.normalized_shape = torch.Size(normalized_shape)
        if len(self.normalized_shape) != 1:
            raise RuntimeError("FusedLayerNorm normalises over the last axis only")
        self.eps = eps
        self._width = int(normalized_shape[0])
        self.register_parameter("weight", Parameter(torch.ones(*normalized_shape)) if create_scale else None)
        self.register_parameter("bias", Parameter(torch.zeros(*normalized_shape)) if create_offset else None)

    def __setstate__(self, state) -> None:
        super().__setstate__(state)
        self._width = int(self.normalized_shape[0])      # modules saved whole before it existed have none

    def reset_parameters(self) -> None:
        if self.weight is not None:
            torch.nn.init.ones_(self.weight)
        if self.bias is not None:
            torch.nn.init.zeros_(self.bias)

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        p = self._parameters            # the attributes by the short way
        try:
            weight, bias = p["weight"], p["bias"]
        except KeyError:                # parametrised, flattened or replicated: a property or a plain attribute
            weight, bias = self.weight, self.bias
        return _layer_norm(input, weight, bias, self._width, self.eps)


def LayerNorm(c_in: int, create_scale: bool = True, create_offset: bool = True, eps: float = 1e-5) -> torch.nn.Module:
    return FusedLayerNorm(c_in, create_scale=create_scale, create_offset=create_offset, eps=eps)
