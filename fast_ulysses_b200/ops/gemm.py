"""bf16 GEMM on the tcgen05 tensor cores (csrc/kernels/gemm_sm100.cu).

``gemm_bf16(a, b)`` computes ``a @ b.T`` with fp32 accumulation in tensor memory; bias, GELU and a
residual add are fused into the epilogue. Both operands must have a contiguous last (K) axis.
``linear`` wraps it as a differentiable ``F.linear``: the backward runs two more of these GEMMs that
read dY, X and W as they lie in memory (``a_km`` / ``b_kn``), so every contraction of the block
stays on this kernel and nothing is transposed or copied. Argument handling and autograd are native
(csrc/ops/fused.cc).
"""

from __future__ import annotations

import torch

from .. import _C


def error_word(device: torch.device) -> torch.Tensor:
    """One device word per GPU that kernels set when one of their bounded waits ran out."""
    return _C.error_word(device.index if device.index is not None else torch.cuda.current_device())


def check_errors(device: torch.device | None = None) -> None:
    """Synchronising: raises if any tcgen05 kernel on this device gave up on a wait."""
    device = device or torch.device("cuda", torch.cuda.current_device())
    code = int(error_word(device).item())
    if code:
        error_word(device).zero_()
        raise RuntimeError(f"fast_ulysses_b200: a tcgen05 kernel gave up on an internal wait (code {code})")


def gemm_bf16(a: torch.Tensor, b: torch.Tensor, *, bias: torch.Tensor | None = None,
              residual: torch.Tensor | None = None, act: int = 0, out: torch.Tensor | None = None,
              ctas: int = 0, a_km: bool = False, b_kn: bool = False, aux: torch.Tensor | None = None,
              store_pre: torch.Tensor | None = None, pair: bool | None = None) -> torch.Tensor:
    """``out[m, n] = act(a[m, :] . b[n, :] + bias[n]) + residual[m, n]`` (bf16 in, bf16 out).

    ``act``: 0 none, 1 GELU (tanh form), 2 GELU (erf form), 3 multiply by the derivative of the
    tanh-form GELU at ``aux[m, n]`` (the activation's backward, fused into the GEMM that produces
    its incoming gradient). ``store_pre`` (m, n) also receives the value before the activation.

    ``a_km`` / ``b_kn``: that operand is given with the contraction along its rows, ``a`` as
    ``(k, m)`` and ``b`` as ``(k, n)``; the kernel reads it as it lies in memory (no transposed
    copy), which is what the weight gradient ``dY^T X`` of a linear layer wants.

    ``ctas``: run on at most that many SMs and leave the others to kernels of other streams.

    ``pair``: run on pairs of CTAs (two 256 x 256 blocks each, one tcgen05 MMA over two SMs) or on
    single CTAs (128 x 128 tiles), with the same bits; ``None`` leaves the shape to the library, which may
    also share K between CTAs and so sum in another order."""
    return _C.gemm_bf16(a, b, bias, residual, act, out, ctas, a_km, b_kn, aux, store_pre, pair)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None,
           residual: torch.Tensor | None = None) -> torch.Tensor:
    """Differentiable ``x @ weight.T + bias (+ residual)`` on the tcgen05 GEMM (bf16); the residual is
    added in the GEMM's epilogue."""
    return _C.linear(x, weight, bias, residual)


def feed_forward(x, w1, b1, w2, b2, residual=None) -> torch.Tensor:
    """``gelu_tanh(x @ w1.T + b1) @ w2.T + b2 (+ residual)``, differentiable, four epilogue-fused GEMMs
    forward + backward-input and two weight-gradient GEMMs; no separate activation or add kernel."""
    return _C.feed_forward(x, w1, b1, w2, b2, residual)
