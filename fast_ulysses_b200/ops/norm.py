"""LayerNorm without affine parameters as one kernel forward and one backward
(csrc/kernels/elementwise.cu: fu_layernorm_fwd / fu_layernorm_bwd_add; autograd in csrc/ops/fused.cc): bf16
in and out, statistics in fp32. The DiT blocks normalise with it so that no eager elementwise kernel
runs between the GEMMs."""

from __future__ import annotations

import torch

from .. import _C


def layer_norm(x: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """``(x - mean) / sqrt(var + eps)`` over the last axis of a bf16 tensor (no weight, no bias)."""
    return _C.layer_norm(x, eps)


def layer_norm_fork(x: torch.Tensor, eps: float = 1e-6) -> tuple[torch.Tensor, torch.Tensor]:
    """``(layer_norm(x), x)`` for a norm in front of a residual branch: the gradients of both results are
    joined inside the norm's backward kernel instead of by an addition of its own."""
    return _C.layer_norm_fork(x, eps)
