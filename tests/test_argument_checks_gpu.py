"""What the differentiable entry points refuse. Each refusal is made on the host, before a kernel starts: an
operand on another device, or one that is shorter than what an epilogue reads, would otherwise be an address
that the kernel may not touch."""

import pytest
import torch
from cuda.bindings import driver

import fast_ulysses_b200 as fu
from fast_ulysses_b200.models.attention import UlyssesSelfAttention
from fast_ulysses_b200.ops import _ckernels as ck
from fast_ulysses_b200.ops import attention, fp8, gemm, norm

pytestmark = pytest.mark.gpu

M, K, N = 24, 64, 40


def bf16(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def short_epilogues(rows, n):
    """Name, bias and residual of a product of ``rows`` x ``n`` that an epilogue must not be given."""
    return [("a bias that is too short", bf16(n - 8), None), ("a bias on the host", bf16(n).cpu(), None),
            ("a residual that would broadcast", None, bf16(1, n)), ("a residual of too few rows", None, bf16(rows - 1, n)),
            ("an fp32 residual", None, torch.randn(rows, n, device="cuda")), ("a residual on the host", None, bf16(rows, n).cpu())]


@pytest.mark.parametrize("train", [False, True])
def test_linear_refuses(train):
    x, w = bf16(2, M // 2, K).requires_grad_(train), bf16(N, K)
    for what, bias, residual in short_epilogues(M, N):
        with pytest.raises(AssertionError):
            gemm.linear(x, w, bias, residual)
            pytest.fail(what)
    with pytest.raises(AssertionError):
        gemm.linear(x, w.cpu())
    # and takes what it always took: a bias of another type or with a leading axis, a flat residual
    for bias in (torch.randn(N, device="cuda"), torch.randn(N, device="cuda").half(), bf16(1, N)):
        assert gemm.linear(x, w, bias, bf16(M, N)).shape == (2, M // 2, N)


@pytest.mark.parametrize("train", [False, True])
def test_feed_forward_refuses(train):
    x, w1, w2 = bf16(2, M // 2, K).requires_grad_(train), bf16(N, K), bf16(K, N)
    good = [x, w1, bf16(N), w2, bf16(K)]
    gemm.feed_forward(*good, residual=bf16(2, M // 2, K))
    for at in (1, 2, 3, 4):  # every weight and bias, left on the host
        args = list(good)
        args[at] = args[at].cpu()
        with pytest.raises(AssertionError):
            gemm.feed_forward(*args)
    with pytest.raises(AssertionError):
        gemm.feed_forward(x, w1, bf16(N - 8), w2, None)
    for what, bias, residual in short_epilogues(M, K):
        with pytest.raises(AssertionError):
            gemm.feed_forward(x, w1, None, w2, bias, residual)
            pytest.fail(what)


@pytest.mark.parametrize("name,value", [("w_qkv", lambda p: p.cpu()), ("w_o", lambda p: p.cpu()), ("b_o", lambda p: p.cpu()),
                                        ("b_o", lambda p: p[:-8]), ("gamma_q", lambda p: p[:64]), ("gamma_k", lambda p: p.cpu())])
def test_attention_block_refuses_a_parameter_it_cannot_read(name, value):
    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(1, 4, 8))
    x = bf16(1, 32, 256)
    assert attn(x, residual=x).shape == x.shape
    setattr(attn, name, torch.nn.Parameter(value(getattr(attn, name).detach())))
    with pytest.raises(AssertionError):
        attn(x, residual=x)
    gemm.check_errors()
    g.check()
    g.destroy()


def test_attention_block_refuses_a_residual_on_the_host():
    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(1, 4, 8))
    x = bf16(1, 32, 256)
    with pytest.raises(AssertionError):
        attn(x, residual=x.cpu())
    g.destroy()


@pytest.mark.parametrize("mode", [torch.enable_grad, torch.no_grad])
def test_forward_mode_tangents_are_refused_and_not_dropped(mode):
    import torch.autograd.forward_ad as fw

    g = fu.UlyssesGroup(device="cuda")
    attn = UlyssesSelfAttention(g, 256, 2, grid=(1, 4, 8))
    q = bf16(1, 32, 2, 128)
    calls = [(lambda t: gemm.linear(t, bf16(N, K)), bf16(M, K)), (lambda t: gemm.linear(bf16(M, K), t), bf16(N, K)),
             (lambda t: gemm.feed_forward(t, bf16(N, K), None, bf16(K, N), None), bf16(M, K)),
             (norm.layer_norm, bf16(M, K)), (norm.layer_norm_fork, bf16(M, K)), (lambda t: attention.attention(q, t, q), bf16(1, 32, 2, 128)),
             (attn, bf16(1, 32, 256))]
    with fw.dual_level(), mode():
        for call, x in calls:
            call(x)
            with pytest.raises(RuntimeError, match="jvp|forward AD"):
                call(fw.make_dual(x, torch.randn_like(x)))
    g.destroy()


def test_attention_refuses_operands_it_cannot_read():
    q, k, v = bf16(2, 30, 3, 128), bf16(2, 50, 3, 128), bf16(2, 50, 3, 128)
    o, lse = attention.fmha_fwd(q, k, v)
    d_o = torch.randn_like(o)
    attention.fmha_bwd(q, k, v, o, lse, d_o)
    for args in ((q, k.cpu(), v), (q, k, v.cpu()), (q, k[:, :, :2], v[:, :, :2]), (q, k[:1], v[:1]), (q, k, v[:, :40])):
        with pytest.raises(AssertionError):
            attention.attention(*args)
        with pytest.raises(AssertionError):
            attention.fmha_bwd(*args, o, lse, d_o)
    with pytest.raises(AssertionError):
        attention.fmha_fwd(q, k, v, out=torch.empty(2, 29, 3, 128, device="cuda", dtype=torch.bfloat16))
    for bad in ((o, lse.cpu(), d_o), (o, lse[:1], d_o), (o, lse.double(), d_o), (o, lse, d_o.cpu()), (o, lse, d_o[:, :20]),
                (o[:, :20], lse, d_o[:, :20])):
        with pytest.raises(AssertionError):
            attention.fmha_bwd(q, k, v, *bad)
    for bad in ((q, k, v[:, :40].contiguous()), (q, k.cpu(), v), (q.float(), k, v)):
        with pytest.raises(AssertionError):
            attention.fmha_bwd(q, k, v, o, lse, d_o, out=tuple(torch.empty_like(t) for t in bad))


@pytest.mark.parametrize("name", ["bias", "residual", "out", "aux", "store_pre"])
def test_gemm_refuses_an_operand_on_the_host(name):
    a, b = bf16(M, K), bf16(N, K)
    extra = {name: torch.zeros(N) if name == "bias" else torch.zeros(M, N).bfloat16()}
    with pytest.raises(AssertionError):
        gemm.gemm_bf16(a, b, **extra)
    with pytest.raises(AssertionError):
        gemm.gemm_bf16(a, b.cpu())
    assert gemm.gemm_bf16(a, b, **{k: v.cuda() for k, v in extra.items()}).shape == (M, N)


def test_a_launch_that_fails_is_reported_once():
    """A stream whose capture has been spoilt refuses the launch; the next call, on another one, is not told of it again."""
    x, y = bf16(24, 128), bf16(24, 128)
    stream = driver.cuStreamCreate(driver.CUstream_flags.CU_STREAM_NON_BLOCKING)[1]
    driver.cuStreamBeginCapture(stream, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED)
    driver.cuStreamSynchronize(stream)  # not allowed while it is captured
    rc = ck.lib().fu_layernorm_fwd(x.data_ptr(), y.data_ptr(), None, 24, 128, 128, 128, 1e-6, int(stream))
    driver.cuStreamEndCapture(stream)
    driver.cuStreamDestroy(stream)
    with pytest.raises(RuntimeError, match="capture"):
        ck.check(rc)
    back = fp8.dequantize(fp8.quantize(x))  # launched in the ordinary way
    assert ((back - x).norm() / x.norm()).item() < 0.04  # three bits of mantissa: 2^-4 at most
