"""``dropout_add_rowwise``: residual + dropout(x) with the dropout mask shared along axis -3.

Mirror of protenix/model/modules/fused_ops.py:190-224.  In eval mode (or p = 0) the op is ``residual + x`` (:213-214);
the fused kernels of this package fold that add into their epilogues, and this function exists for API compatibility.
In training mode the mask of shape [..., 1, C, D] is drawn exactly as the reference's own fallback draws it
(``dropout`` of a tensor of ones, :219-223), so the same seed gives the same mask, and the scaled product and the add
run in one kernel (``px_scale_add_rowwise``), forward and backward.  CUDA tensors only.
"""
import torch

from . import native


def dropout_add_rowwise(residual: torch.Tensor, x: torch.Tensor, p_drop: float, training: bool) -> torch.Tensor:
    if not training or p_drop == 0.0:
        return residual + x
    if not x.is_cuda:
        raise RuntimeError("dropout_add_rowwise (training): CUDA tensors only, this package has no CPU path")
    return native.load().dropout_add(residual, x, p_drop)
