"""The fused sequence-parallel attention block and the DiT stack on ONE GPU (a single-rank group
runs every fused kernel: scatter epilogue, attention, pull prologue) against plain PyTorch."""

import pytest
import torch

import fast_ulysses_b200 as fu
from fast_ulysses_b200.models.attention import UlyssesSelfAttention, reference_attention
from fast_ulysses_b200.models.dit import DiTBlock, DiTStack, reference_forward
from fast_ulysses_b200.ops import gemm

pytestmark = pytest.mark.gpu


def rel_err(got, want):
    return ((got.float() - want.float()).norm() / want.float().norm().clamp_min(1e-12)).item()


def test_attention_block_forward_backward_single_rank():
    torch.manual_seed(0)
    g = fu.UlyssesGroup(device="cuda")
    grid, hidden, heads = (3, 10, 16), 512, 4  # 480 tokens
    attn = UlyssesSelfAttention(g, hidden, heads, grid=grid)
    with torch.no_grad():
        attn.gamma_q.add_(0.1 * torch.randn_like(attn.gamma_q))
        attn.gamma_k.add_(0.1 * torch.randn_like(attn.gamma_k))
        attn.b_o.add_(0.1 * torch.randn_like(attn.b_o.float()).bfloat16())
    x = torch.randn(1, 480, hidden, device="cuda").bfloat16().requires_grad_()
    y = attn(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    gemm.check_errors()
    g.check()

    params = [attn.w_qkv, attn.gamma_q, attn.gamma_k, attn.w_o, attn.b_o]
    xr = x.detach().float().requires_grad_()
    pr = [p.detach().float().requires_grad_() for p in params]
    yr = reference_attention(xr, pr[0], pr[1], pr[2], pr[3], pr[4], heads, grid)
    yr.backward(dy.float())
    assert rel_err(y, yr) < 2e-2, rel_err(y, yr)
    assert rel_err(x.grad, xr.grad) < 3e-2, ("dx", rel_err(x.grad, xr.grad))
    for name, p, r in zip(("w_qkv", "gamma_q", "gamma_k", "w_o", "b_o"), params, pr):
        assert rel_err(p.grad, r.grad) < 4e-2, (name, rel_err(p.grad, r.grad))
    g.destroy()


def test_dit_stack_single_rank():
    torch.manual_seed(1)
    g = fu.UlyssesGroup(device="cuda")
    grid = (2, 8, 16)  # 256 tokens
    stack = DiTStack(g, depth=2, hidden=256, heads=2, ffn=512, grid=grid)
    x = torch.randn(1, 256, 256, device="cuda").bfloat16().requires_grad_()
    y = stack(x)
    y.float().pow(2).mean().backward()
    gemm.check_errors()
    xr = x.detach().float().requires_grad_()
    yr = reference_forward(stack, xr)
    yr.pow(2).mean().backward()
    assert rel_err(y, yr) < 3e-2, rel_err(y, yr)
    assert rel_err(x.grad, xr.grad) < 6e-2, rel_err(x.grad, xr.grad)
    g.destroy()


def test_backward_after_a_later_forward_is_refused():
    """The block keeps q, k, v and the attention output in its symmetric buffers: a backward for a
    forward that a later forward has overwritten must raise, not return another call's gradients."""
    torch.manual_seed(2)
    g = fu.UlyssesGroup(device="cuda")
    grid, hidden, heads = (2, 8, 16), 256, 2
    attn = UlyssesSelfAttention(g, hidden, heads, grid=grid)
    x1 = torch.randn(1, 256, hidden, device="cuda").bfloat16().requires_grad_()
    x2 = torch.randn(1, 256, hidden, device="cuda").bfloat16().requires_grad_()
    y1 = attn(x1)
    y2 = attn(x2)
    with pytest.raises(RuntimeError, match="forward ran again"):
        y1.sum().backward()
    y2.sum().backward()  # the latest forward still owns the buffers
    # forward, backward, forward, backward (gradient accumulation) is the supported order
    attn.zero_grad()
    attn(x1).sum().backward()
    first = attn.w_o.grad.clone()
    attn(x1).sum().backward()
    assert torch.allclose(attn.w_o.grad.float(), 2 * first.float(), rtol=2e-2, atol=1e-3)
    gemm.check_errors()
    g.destroy()


def test_norm_weights_may_be_slices_of_a_flat_buffer():
    """Parameters kept in one flat buffer start on any element, not on the 16 bytes a vector load needs."""
    torch.manual_seed(3)
    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(2, 4, 8))
    x = torch.randn(1, 64, 256, device="cuda").bfloat16()
    dy = torch.randn_like(x)
    flat = torch.rand(3 + 2 * 129, device="cuda") + 0.5
    grads = []
    for at in (3, 4):  # 4: 16-byte aligned slices of the same values
        flat[at:at + 128] = torch.linspace(0.5, 1.5, 128, device="cuda")
        flat[at + 128:at + 256] = torch.linspace(1.5, 0.5, 128, device="cuda")
        attn.gamma_q = torch.nn.Parameter(flat[at:at + 128])
        attn.gamma_k = torch.nn.Parameter(flat[at + 128:at + 256])
        attn.w_qkv.grad = None
        y = attn(x)
        y.backward(dy)
        grads.append((y.detach(), attn.w_qkv.grad, attn.gamma_q.grad, attn.gamma_k.grad))
    gemm.check_errors()
    for name, a, b in zip(("y", "w_qkv", "gamma_q", "gamma_k"), *grads):
        # dq and d(gamma) are summed in fp32 in another order from call to call
        assert rel_err(a, b) < 2e-3, name
    g.destroy()


def test_block_takes_a_gradient_that_starts_anywhere():
    """The gradient of the result is also that of the second half's residual: a dense tensor at an odd offset of a
    larger buffer is no different from its copy. Nor is such a residual of the attention block."""
    torch.manual_seed(4)
    g = fu.UlyssesGroup(device="cuda")
    block = DiTBlock(g, 256, 2, 512, grid=(2, 4, 8))
    x = torch.randn(1, 64, 256, device="cuda").bfloat16().requires_grad_()
    odd = torch.randn(64 * 256 + 3, device="cuda").bfloat16()[3:].view(1, 64, 256)
    grads = []
    for dy in (odd, odd.clone()):
        x.grad = None
        block(x).backward(dy)
        grads.append(x.grad)
    assert rel_err(*grads) < 2e-3  # dq is summed in fp32 in another order from call to call
    with torch.no_grad():
        assert torch.equal(block.attn(x, residual=odd), block.attn(x, residual=odd.clone()))
    gemm.check_errors()
    g.destroy()


def test_bf16_norm_weights_written_through_data_are_seen():
    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(2, 4, 8))
    attn.gamma_q = torch.nn.Parameter(attn.gamma_q.detach().bfloat16())
    x = torch.randn(1, 64, 256, device="cuda").bfloat16()
    dy = torch.randn_like(x)
    for value in (1.0, 3.0):
        attn.gamma_q.data.fill_(value)  # as an optimizer that keeps fp32 master weights does
        attn.zero_grad()
        y = attn(x)
        y.backward(dy)
        got = y.detach(), attn.gamma_k.grad
        attn.gamma_q = torch.nn.Parameter(torch.full((128,), value, device="cuda", dtype=torch.bfloat16))
        attn.zero_grad()
        fresh = attn(x)
        fresh.backward(dy)
        assert torch.equal(got[0], fresh)
        assert rel_err(got[1], attn.gamma_k.grad) < 1e-4  # summed in fp32 in another order from call to call
    g.destroy()


def test_eps_and_timeout_set_later_take_effect():
    torch.manual_seed(6)
    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(2, 4, 8), eps=1e-6, timeout_ms=700)
    x = torch.randn(1, 64, 256, device="cuda").bfloat16()
    with torch.no_grad():
        before = attn(x)
        attn.eps, attn.timeout_ms = 0.5, 900
        after = attn(x)
        want = reference_attention(x, attn.w_qkv, attn.gamma_q, attn.gamma_k, attn.w_o, attn.b_o, 2, (2, 4, 8), eps=0.5)
    assert not torch.equal(before, after) and rel_err(after, want) < 2e-2
    assert (attn.eps, attn.timeout_ms, attn._native.timeout_ms) == (0.5, 900, 900)
    g.destroy()
