"""Flash attention on the tcgen05 tensor cores (csrc/kernels/fmha_fwd_sm100.cu, fmha_bwd_sm100.cu;
argument handling and autograd in csrc/ops/fused.cc).

Tensors use the ``(batch, seq, heads, 128)`` layout of the all-to-all windows; any view whose last
axis is contiguous and whose other strides are multiples of 8 elements is read in place.
"""

from __future__ import annotations

import math

import torch

from .. import _C
from .gemm import error_word


def _strides(t: torch.Tensor):
    assert t.dim() == 4 and t.shape[-1] == 128 and t.stride(3) == 1 and t.dtype == torch.bfloat16, (t.shape, t.stride())
    return t.stride(1), t.stride(2), t.stride(0)


def _fill(a, q, k, v, o):
    """Operands, shape and strides of a ``_ckernels.FuFmhaArgs`` for a caller of the C symbols themselves."""
    b, sq, h, _ = q.shape
    a.q, a.k, a.v, a.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr()
    a.batch, a.heads, a.seq_q, a.seq_kv, a.head_dim = b, h, sq, k.shape[1], 128
    a.q_row, a.q_head, a.q_batch = _strides(q)
    a.k_row, a.k_head, a.k_batch = _strides(k)
    a.v_row, a.v_head, a.v_batch = _strides(v)
    a.o_row, a.o_head, a.o_batch = _strides(o)
    a.err = error_word(q.device).data_ptr()


def fmha_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: float | None = None,
             out: torch.Tensor | None = None, ctas: int = 0, poly: int | None = None,
             trace: torch.Tensor | None = None):
    """``softmax(q k^T * scale) v`` for (b, s, h, 128) bf16 tensors. Returns ``(o, lse)`` with
    ``lse`` of shape (b, h, s_q), fp32, natural log. ``poly`` (0, 2, 4 or 6) overrides how many of
    every 16 exponential pairs are computed on the FMA pipe instead of the special-function unit.
    ``trace`` (int64[256] on the device) selects the instrumented build of the kernel: CTA 0 stores the
    SM clock of 32 pipeline events for kv steps 64..71 of its first item."""
    flags = 0 if poly is None else 0x1000 | ((poly & 15) << 8)  # FU_FMHA_POLY(poly)
    return _C.fmha_fwd(q, k, v, scale, out, ctas, flags, trace)


def attention_reference(q, k, v, scale=None):
    """fp32 PyTorch statement on (b, s, h, d) tensors; returns (o, lse)."""
    scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * scale
    lse = torch.logsumexp(s, dim=-1)
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, dim=-1), v.float())
    return o, lse


def fmha_bwd(q, k, v, o, lse, d_o, *, scale: float | None = None, ctas: int = 0, out=None,
             deterministic: bool = False, trace: torch.Tensor | None = None):
    """Gradients of ``fmha_fwd``. All tensors (b, s, h, 128) bf16; ``d_o`` must share ``o``'s
    strides. Returns ``(dq, dk, dv)`` shaped and strided like q, k, v (dense). The default is one
    software-pipelined pass that sums dQ over the K/V blocks with fp32 reductions (dK and dV are
    bit-reproducible, dQ to rounding); ``deterministic=True`` runs two passes without atomics
    (dK/dV with the K/V block stationary, then dQ with the query rows stationary) at about 2.4x
    the time."""
    return _C.fmha_bwd(q, k, v, o, lse, d_o, scale, ctas, None if out is None else list(out), deterministic, trace)


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float | None = None) -> torch.Tensor:
    """Differentiable non-causal attention on (b, s, h, 128) bf16 tensors (tcgen05 fwd and bwd)."""
    return _C.attention(q, k, v, scale)
