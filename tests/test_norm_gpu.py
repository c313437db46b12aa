"""The one-kernel LayerNorm (forward and backward) against PyTorch in fp32."""

import pytest
import torch

from fast_ulysses_b200.ops.norm import layer_norm, layer_norm_fork

pytestmark = pytest.mark.gpu


def rel_err(got, want):
    return ((got.float() - want.float()).norm() / want.float().norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("shape", [(1, 37, 256), (2, 130, 5120), (3, 8)])
def test_layer_norm_forward_and_backward(shape):
    torch.manual_seed(sum(shape))
    x = (torch.randn(*shape, device="cuda") * 3 + 1.5).bfloat16().requires_grad_()
    y = layer_norm(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr = x.detach().float().requires_grad_()
    yr = torch.nn.functional.layer_norm(xr, (shape[-1],), eps=1e-6)
    yr.backward(dy.float())
    assert rel_err(y, yr) < 1e-2, rel_err(y, yr)
    assert rel_err(x.grad, xr.grad) < 1.5e-2, rel_err(x.grad, xr.grad)


def test_layer_norm_reads_a_row_strided_view_in_place():
    torch.manual_seed(1)
    big = torch.randn(64, 512, device="cuda").bfloat16()
    x = big[:, :256]  # rows 1024 bytes apart, 512 bytes used
    y = layer_norm(x)
    want = torch.nn.functional.layer_norm(x.float(), (256,), eps=1e-6)
    assert rel_err(y, want) < 1e-2


# one unit a lane to five with one warp a row, the last column beyond; the same with two, four and eight warps; rows that are
# walked through; a matrix beyond L2; last CTAs with rows missing
@pytest.mark.parametrize("rows, cols", [(1, 8), (9, 256), (7, 264), (17, 1280), (3, 1288), (5, 2560), (3, 2568), (7, 5120), (3, 5128), (2, 10240),
                                        (3, 10248), (2, 20000), (2501, 5120), (9831, 1288)])
def test_layer_norm_rows_of_every_form(rows, cols):
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    x, g, r = (torch.randn(rows, cols, device="cuda", generator=gen).mul_(2).add_(0.5).bfloat16() for _ in range(3))
    x.requires_grad_()
    y, past = layer_norm_fork(x)
    torch.autograd.backward((y, past), (g, r))
    xr = x.detach().double().requires_grad_()
    yr = torch.nn.functional.layer_norm(xr, (cols,), eps=1e-6)
    torch.autograd.backward((yr, xr * 1), (g.double(), r.double()))
    for got, want in ((y.detach(), yr.detach()), (x.grad, xr.grad)):
        # one rounding to bf16 (2^-9 of the value) and fp32 sums of values of a few units
        assert ((got.double() - want).abs() <= 2**-8 * want.abs() + 1e-4).all()


# beyond L2: in registers without a gradient to add, with one walked through, rows of one unit too
@pytest.mark.parametrize("rows, cols", [(50001, 256), (9831, 1288), (2501, 5120), (1301, 10240)])
@pytest.mark.parametrize("fork", [False, True])
def test_layer_norm_backward_beyond_l2(rows, cols, fork):
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    x, g, r = (torch.randn(rows, cols, device="cuda", generator=gen).bfloat16() for _ in range(3))
    x.requires_grad_()
    if fork:
        torch.autograd.backward(layer_norm_fork(x), (g, r))
    else:
        layer_norm(x).backward(g)
    xr = x.detach().double().requires_grad_()
    torch.nn.functional.layer_norm(xr, (cols,), eps=1e-6).backward(g.double())
    want = xr.grad + r.double() if fork else xr.grad
    # one rounding to bf16 (2^-9 of the value) and fp32 sums of values of a few units
    assert ((x.grad.double() - want).abs() <= 2**-8 * want.abs() + 1e-4).all()


# a mean that has overflowed: -inf in every column, whether or not the row fills its lanes
@pytest.mark.parametrize("cols", [256, 264, 1288, 5128, 10248])
def test_layer_norm_backward_of_an_overflowed_mean(cols):
    x = torch.full((3, cols), 3e38, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = layer_norm(x)
    y.backward(torch.ones_like(y))
    assert (x.grad == float("-inf")).all()


def _shortest(call, runs=9, calls=4):
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(runs):
        start.record()
        for _ in range(calls):
            call()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times)


# the shortest rows of two and of four warps: bound by HBM, as a copy is (1.0 - 1.1 times its time; with a row's number of warps
# unknown to the compiler 1.3 - 1.4)
@pytest.mark.parametrize("cols", [1288, 2568])
def test_layer_norm_of_large_matrices_takes_what_a_copy_takes(cols):
    x = torch.randn(75600, cols, device="cuda", dtype=torch.bfloat16)
    y = torch.empty_like(x)
    for call in (lambda: y.copy_(x), lambda: layer_norm(x)):
        call()
    assert _shortest(lambda: layer_norm(x)) < 1.22 * _shortest(lambda: y.copy_(x))
