"""What is kept of parameters between calls: when it is renewed, and the 16-bit copies of the tensor wrappers.

The kernels consume 16-bit weight matrices: bf16 where the weight multiplies rows of a bf16 pair tensor, fp16
where it multiplies fp16 operands (rows of an fp32 pair tensor, which the kernels standardise and round to fp16,
and every intermediate tensor).  The modules keep fp32 parameters with the reference's names so that its
checkpoints load with ``strict=True``.  A cached copy is keyed on the parameter's storage pointer, device, in-place
version counter and the wanted format, so ``load_state_dict``, ``.to()`` and optimiser steps all invalidate it.
Inside a CUDA graph capture nothing is looked up or kept: the conversion becomes part of the graph.  A stream that uses a
copy for the first time waits for its conversion, and the copy's memory is not given out again before that stream is through with it.

The modules keep laid-out weights in the same way (``native.py``).  Both see new parameter objects, new storages and every write
that PyTorch counts as an in-place change (``tensor._version``).  A write past that counter, as ``p.data.copy_(ema)`` or a kernel
that was given the address, is not seen: ``weights_changed(module)`` announces it.
"""
from __future__ import annotations

import weakref
from typing import Dict, Tuple

import torch
from torch.multiprocessing.reductions import StorageWeakRef


class _Copy:
    """One kept copy: of which state of which parameter, and the streams that may use it without further ado."""

    def __init__(self, key: Tuple, w: torch.Tensor, ref: "weakref.ref", storage: StorageWeakRef) -> None:
        self.key, self.w, self.ref, self.storage = key, w, ref, storage
        if w.is_cuda:
            stream = torch.cuda.current_stream(w.device)
            self.made, self.streams = stream.record_event(), {stream.cuda_stream}

    def for_current_stream(self) -> torch.Tensor:
        if self.w.is_cuda:
            stream = torch.cuda.current_stream(self.w.device)
            if stream.cuda_stream not in self.streams:
                stream.wait_event(self.made)
                self.w.record_stream(stream)
                self.streams.add(stream.cuda_stream)
        return self.w


_cache: Dict[Tuple[int, torch.dtype], _Copy] = {}


def w16_of(p: torch.Tensor, fmt: torch.dtype) -> torch.Tensor:
    """``p`` as a contiguous tensor of the 16-bit format ``fmt`` (``torch.bfloat16`` or ``torch.float16``)."""
    if p.dtype == fmt and p.is_contiguous() and not p.requires_grad:
        return p
    if p.is_cuda and torch.cuda.is_current_stream_capturing():
        return p.detach().to(fmt).contiguous()       # written by the graph's replays, into the graph's own memory
    storage = p.untyped_storage()       # held weakly: another storage has another address, also where its memory lies where the old one's did
    key = (p.data_ptr(), storage._cdata, p._version, p.device, tuple(p.shape), p.dtype)
    ent = _cache.get((id(p), fmt))
    if ent is not None and ent.key == key and ent.ref() is p:
        return ent.for_current_stream()
    w = p.detach().to(fmt).contiguous()
    ck = (id(p), fmt)
    _cache[ck] = _Copy(key, w, weakref.ref(p, lambda _r, ck=ck: _cache.pop(ck, None)), StorageWeakRef(storage))
    return w


def bf16_of(p: torch.Tensor) -> torch.Tensor:
    return w16_of(p, torch.bfloat16)


def f16_of(p: torch.Tensor) -> torch.Tensor:
    return w16_of(p, torch.float16)


def clear() -> None:
    _cache.clear()


def weights_changed(module: torch.nn.Module) -> None:
    """Says that the weights of ``module`` may have been written past their version counters: everything kept of them is renewed on the
    next call, by whichever module keeps it.  Needed after ``p.data.copy_(...)`` and the like only."""
    torch.autograd.graph.increment_version(
        [t for m in module.modules() for t in [*m.parameters(recurse=False), *m.buffers(recurse=False), *m.__dict__.values()]
         if isinstance(t, torch.Tensor)])
