"""Sequence-parallel self-attention for video DiT blocks, built from the fused sm_100a kernels.

Forward (three kernels, no separate exchange, no permute, no staging copy):
  1. ``fu_qkv_rope_scatter``  x W_qkv^T -> per-head RMSNorm -> 3D RoPE -> every head-row stored
     straight into the owning rank's q/k/v window (mode 0 of the all-to-all is the store address)
  2. ``fu_fmha_fwd``          tcgen05 flash attention reading q/k/v from the window, writing the
     attention output into a symmetric buffer
  3. ``fu_pull_outproj``      the output projection pulls its A operand from the peers' attention
     outputs tile by tile (mode 1 of the all-to-all is the load address)
Backward mirrors it: the gradient of the attention output is scattered to the head owners from
the epilogue of the dgrad GEMM (same kernel as 1 without norm/RoPE, reading W_o as stored),
tcgen05 flash attention backward writes dq/dk/dv into a symmetric buffer, and ONE kernel
(``fu_pull_qkv_grads``) pulls them home from the head owners over NVLink while undoing RoPE and
RMSNorm on the way and writes the operand of the dgrad/wgrad GEMMs: no stand-alone exchange, no
separate norm/RoPE backward, no slice copy, no transposed weight.

The reference ships no model code; its example (examples/dit_attention.py:21-63) wraps nn.Linear
and torch SDPA around two all_to_all_4d calls. ``reference_attention`` below is that composition,
used as the oracle.
"""

from __future__ import annotations

import math

import torch
import torch.nn as nn

from .. import _C
from ..ops.rope import apply_rope_reference, rope_table

HEAD_DIM = 128


class SymmBuffer:
    """A caller-owned symmetric byte buffer plus its address on every rank."""

    def __init__(self, group, nbytes: int):
        nbytes = (nbytes + 255) // 256 * 256
        self.tensor = group._handle.symm_alloc(nbytes)
        ptrs = group._handle.symm_ptrs(self.tensor)
        w = group.world_size
        self.base, self.ctrl = list(ptrs[:w]), list(ptrs[w:])
        self.nbytes = nbytes

    def view(self, offset: int, shape, dtype=torch.bfloat16) -> torch.Tensor:
        n = math.prod(shape) * torch.empty((), dtype=dtype).element_size()
        return self.tensor[offset:offset + n].view(dtype).view(*shape)


class UlyssesSelfAttention(nn.Module):
    """Self-attention over a sequence sharded across ``group`` (Ulysses), Wan2.1-style: fused QKV
    projection, per-head RMSNorm on q and k, 3D RoPE, non-causal attention, output projection.

    Construction is collective (it allocates symmetric buffers). ``seq_splits`` / ``head_splits``
    give every rank's shard (default: even). Input ``(b, s_local, hidden)`` bf16.
    """

    def __init__(self, group, hidden: int = 5120, heads: int = 40, *, grid=(21, 45, 80), batch: int = 1,
                 seq_splits: list[int] | None = None, head_splits: list[int] | None = None, eps: float = 1e-6,
                 out_bias: bool = True, timeout_ms: int = 10000):
        super().__init__()
        self.group, self.hidden, self.heads, self.grid = group, hidden, heads, grid
        self.rank, self.world = group.rank, group.world_size
        total = grid[0] * grid[1] * grid[2]
        if seq_splits is None:
            assert total % self.world == 0, "pass seq_splits for a sequence that does not divide"
            seq_splits = [total // self.world] * self.world
        if head_splits is None:
            assert heads % self.world == 0, "pass head_splits for a head count that does not divide"
            head_splits = [heads // self.world] * self.world
        assert sum(seq_splits) == total and sum(head_splits) == heads
        self.seq_splits, self.head_splits = list(seq_splits), list(head_splits)
        self.s_total, self.s_local = total, seq_splits[self.rank]
        self.seq_off = sum(seq_splits[: self.rank])
        self.n_local = head_splits[self.rank]
        self.batch = batch
        dev = group.device

        self.w_qkv = nn.Parameter(torch.randn(3 * heads * HEAD_DIM, hidden, device=dev).mul_(0.02).bfloat16())
        self.w_o = nn.Parameter(torch.randn(hidden, heads * HEAD_DIM, device=dev).mul_(0.02).bfloat16())
        self.b_o = nn.Parameter(torch.zeros(hidden, device=dev).bfloat16()) if out_bias else None
        self.gamma_q = nn.Parameter(torch.ones(HEAD_DIM, device=dev))
        self.gamma_k = nn.Parameter(torch.ones(HEAD_DIM, device=dev))
        self.register_buffer("rope", rope_table(torch.arange(self.seq_off, self.seq_off + self.s_local, device=dev),
                                                grid=grid), persistent=False)

        # Symmetric buffers. Every rank sizes them for the LARGEST head shard, so that offsets agree.
        region = batch * total * max(head_splits) * HEAD_DIM * 2
        region = (region + 255) // 256 * 256
        self._region = region
        self.qkv_win = SymmBuffer(group, 3 * region)
        self.o_buf = SymmBuffer(group, region)
        self.do_win = SymmBuffer(group, region)
        self.dqkv_buf = SymmBuffer(group, 3 * region)  # dq | dk | dv of this rank's heads, pulled by the token owners
        shape = (batch, total, self.n_local, HEAD_DIM)
        self.q_view = self.qkv_win.view(0, shape)
        self.k_view = self.qkv_win.view(region, shape)
        self.v_view = self.qkv_win.view(2 * region, shape)
        self.o_view = self.o_buf.view(0, shape)
        self.do_view = self.do_win.view(0, shape)
        self.dq_view = self.dqkv_buf.view(0, shape)
        self.dk_view = self.dqkv_buf.view(region, shape)
        self.dv_view = self.dqkv_buf.view(2 * region, shape)
        # the same geometry and addresses for the native forward and backward (csrc/ops/fused.cc)
        n = _C.SpAttention()
        n.heads, n.rank, n.world, n.batch, n.region = heads, self.rank, self.world, batch, region
        n.s_local, n.seq_off, n.s_total, n.head_splits = self.s_local, self.seq_off, self.s_total, self.head_splits
        n.timeout_ms, n.eps = timeout_ms, eps
        comm = getattr(group, "_comm_stream", None)
        n.comm_stream = comm.cuda_stream if comm is not None else 0
        n.set_buffers([a for buf in (self.qkv_win, self.o_buf, self.do_win, self.dqkv_buf) for a in (buf.base, buf.ctrl)],
                      [self.q_view, self.k_view, self.v_view, self.o_view, self.do_view, self.dq_view, self.dk_view,
                       self.dv_view])
        self._native = n

    @property
    def eps(self) -> float:
        return self._native.eps

    @eps.setter
    def eps(self, value: float) -> None:
        self._native.eps = value

    @property
    def timeout_ms(self) -> int:
        return self._native.timeout_ms

    @timeout_ms.setter
    def timeout_ms(self, value: int) -> None:
        self._native.timeout_ms = int(value)

    def forward(self, x: torch.Tensor, residual: torch.Tensor | None = None) -> torch.Tensor:
        """``residual`` (same shape as the result) is added in the output projection's epilogue."""
        return _C.sp_attention(self._native, x, self.w_qkv, self.gamma_q, self.gamma_k, self.w_o, self.b_o, residual, self.rope)


def reference_attention(x_full, w_qkv, gamma_q, gamma_k, w_o, b_o, heads, grid, eps=1e-6, compute=torch.float32):
    """The same block without sequence parallelism, in plain PyTorch on the FULL sequence
    (b, S, hidden): linear -> per-head RMSNorm -> RoPE -> SDPA -> linear."""
    b, S, hidden = x_full.shape
    xf = x_full.to(compute)
    y = xf @ w_qkv.to(compute).t()
    q, k, v = (t.reshape(b, S, heads, HEAD_DIM) for t in y.chunk(3, dim=-1))

    def norm(t, g):
        return t * torch.rsqrt(t.float().pow(2).mean(-1, keepdim=True) + eps).to(t.dtype) * g.to(t.dtype)

    table = rope_table(torch.arange(S, device=x_full.device), grid=grid)
    q = apply_rope_reference(norm(q, gamma_q), table).to(compute)
    k = apply_rope_reference(norm(k, gamma_k), table).to(compute)
    o = torch.nn.functional.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2))
    o = o.transpose(1, 2).reshape(b, S, heads * HEAD_DIM)
    out = o @ w_o.to(compute).t()
    return out + b_o.to(compute) if b_o is not None else out
