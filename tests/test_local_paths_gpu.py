"""The single-rank paths and the small kernels beside the GEMMs, at the sizes where they can go wrong:
vector widths, remainders of a CTA's share, the switch between the two launch shapes, ragged rows and
columns. Oracles: plain PyTorch in fp32, or the input itself where bytes are moved."""

import ctypes as C

import pytest
import torch

import fast_ulysses_b200 as fu
from fast_ulysses_b200.ops import _ckernels as ck
from fast_ulysses_b200.ops import fp8, norm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def group():
    g = fu.UlyssesGroup(device="cuda")
    yield g
    g.check()
    g.destroy()


@pytest.mark.parametrize("b,s,n,d,dtype", [
    (1, 1, 1, 8, torch.float16),        # one 16-byte vector
    (1, 3, 1, 8, torch.bfloat16),       # 48 bytes: not a multiple of 32
    (2, 33, 3, 72, torch.bfloat16),     # ragged rows
    (1, 1024, 64, 64, torch.bfloat16),  # 8 MiB: the last size of the small launch shape
    (1, 1025, 64, 64, torch.bfloat16),  # and the first of the large one
    (3, 1111, 13, 80, torch.float32),
])
@pytest.mark.parametrize("layout", ["dense", "packed", "packed_batch", "offset16"])
def test_exchange_of_a_single_rank_moves_every_byte(group, b, s, n, d, dtype, layout):
    gen = torch.Generator(device="cuda").manual_seed(s)
    if layout == "packed":  # pitched rows; batches fold into rows
        x = torch.randn(b, s, 3, n, d, device="cuda", generator=gen).to(dtype)[:, :, 1]
    elif layout == "packed_batch":  # a batch stride that does not fold
        x = torch.randn(b, s + 2, 2, n, d, device="cuda", generator=gen).to(dtype)[:, 1:s + 1, 1]
    elif layout == "offset16":  # 16-byte but not 32-byte aligned
        e = 16 // torch.empty((), dtype=dtype).element_size()
        x = torch.randn(b * s * n * d + e, device="cuda", generator=gen).to(dtype)[e:].view(b, s, n, d)
    else:
        x = torch.randn(b, s, n, d, device="cuda", generator=gen).to(dtype)
    for mode in (0, 1):
        y = group.all_to_all_4d(x, mode=mode)
        assert torch.equal(y, x)
        out = group.empty_output(x, mode=mode)
        assert torch.equal(group.all_to_all_4d(x, mode=mode, out=out), x)


def test_staged_async_call_protects_its_input_and_orders_its_output(group):
    x = torch.randn(1, 4000, 40, 128, device="cuda").bfloat16()
    keep = x.clone()
    out = group.empty_output(x)
    for i in range(20):
        h = group.all_to_all_4d_async(x, out=out)
        x.fill_(float(i))  # the call returned: its input is free
        assert torch.equal(h.wait(), keep)
        x.copy_(keep)
    plain = group.all_to_all_4d_async(x)
    x.zero_()
    assert torch.equal(plain.wait(), keep)


def test_async_call_is_seen_by_dispatch_modes_and_refused_by_vmap(group):
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Recorder(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    x = torch.randn(2, 16, 4, 64, device="cuda").bfloat16()
    out = group.empty_output(x)
    with Recorder():
        y = group.all_to_all_4d_async(x)
        z = group.all_to_all_4d_async(x, out=out, stage=False)
    assert torch.equal(y.wait(), x) and torch.equal(z.wait(), x)
    assert any("all_to_all_4d_staged.default" in s for s in seen) and any("all_to_all_4d_staged_out.default" in s for s in seen)
    with pytest.raises(RuntimeError, match="does not support torch.vmap"):
        torch.vmap(lambda t: group.all_to_all_4d_async(t).wait())(x.unsqueeze(0))


@pytest.mark.parametrize("mode", [0, 1])
def test_staged_async_call_may_write_over_its_input(group, mode):
    buf = group.empty_output(torch.empty(2, 3000, 8, 64, device="cuda", dtype=torch.bfloat16), mode=mode)
    plain = torch.empty_like(buf)
    want = torch.randn(2, 3000, 8, 64, device="cuda").bfloat16()
    for out in (buf, plain):  # a symmetric buffer that the call writes directly, and an ordinary tensor
        out.copy_(want)
        assert torch.equal(group.all_to_all_4d_async(out, mode=mode, out=out).wait(), want)
    packed = torch.randn(2, 3000, 3, 8, 64, device="cuda").bfloat16()
    want = packed[:, :, 1].clone()
    out = packed.view(-1)[:want.numel()].view_as(want)  # overlaps the view it is filled from, row for other row
    assert torch.equal(group.all_to_all_4d_async(packed[:, :, 1], mode=mode, out=out).wait(), want)


@pytest.mark.parametrize("rows", [1, 31, 64, 65, 1000])
def test_fp8_exchange_of_a_single_rank_is_quantise_and_dequantise(group, rows):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(1, rows, 1, 128, device="cuda", generator=gen) * 5).bfloat16()
    x[0, rows // 2] = 0  # an all-zero row keeps scale 1
    assert torch.equal(fp8.all_to_all_4d_fp8(group, x), fp8.dequantize(fp8.quantize(x)))


@pytest.mark.parametrize("rows,cols,pitch", [(1, 8, 8), (3, 5, 5), (255, 64, 64), (256, 72, 80), (4097, 136, 136), (1025, 5120, 5120), (1024, 1024, 1024), (1024, 1025, 1032)])
def test_column_sums(rows, cols, pitch):
    x = torch.randn(rows, pitch, device="cuda").bfloat16()[:, :cols]
    out = torch.empty(cols, device="cuda", dtype=torch.bfloat16)
    fn = ck.lib().fu_colsum_bf16
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int64, C.c_int64, C.c_void_p]
    ck.check(fn(x.data_ptr(), out.data_ptr(), rows, cols, pitch, ck.stream_ptr()))
    want = x.double().sum(0)
    # fp32 sums of `rows` terms, then one rounding to bf16 (relative 2^-9)
    bound = 2.0 ** -8 * want.abs() + rows * 2.0 ** -23 * x.double().abs().sum(0)
    assert torch.all((out.double() - want).abs() <= bound)


@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 264), (300, 5120)])
def test_layer_norm_fork_joins_both_gradients(rows, cols):
    x = torch.randn(rows, cols, device="cuda").bfloat16().requires_grad_()
    gy, gr = torch.randn_like(x), torch.randn_like(x)
    y, r = norm.layer_norm_fork(x)
    assert torch.equal(r, x) and torch.equal(y, norm.layer_norm(x.detach()))
    torch.autograd.backward((y, r), (gy, gr))
    xr = x.detach().double().requires_grad_()
    yr = torch.nn.functional.layer_norm(xr, (cols,), eps=1e-6)
    torch.autograd.backward((yr, xr * 1.0), (gy.double(), gr.double()))
    # one bf16 rounding of a sum of terms of order one
    assert ((x.grad.double() - xr.grad).norm() / xr.grad.norm()).item() < 4e-3
    x.grad = None
    norm.layer_norm_fork(x)[1].backward(gr)  # only the residual is used
    assert torch.equal(x.grad, gr)


def test_first_call_of_a_process_inside_a_graph_capture():
    """Nothing an operator sets up on its first call is refused, or recorded, by a capture."""
    import pathlib
    import subprocess
    import sys

    code = """
import torch
from fast_ulysses_b200.ops import attention, gemm, norm
x = torch.randn(1, 256, 512, device="cuda").bfloat16()
w = torch.randn(512, 512, device="cuda").bfloat16()

def step():
    h = norm.layer_norm(x)
    q = gemm.linear(h, w).view(1, 256, 4, 128)
    return attention.attention(q, q, q)

graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = step()
gemm.check_errors()
graph.replay()
gemm.check_errors()
assert torch.equal(y, step())
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=pathlib.Path(__file__).parents[1])
