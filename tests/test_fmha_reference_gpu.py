"""The forward's exponentials are taken against a loose reference, the first step's maximum, that moves only when a
row's scores leave its range: scores that leave it in any quarter of a kv step, in the first step or later,
by a little or by hundreds of powers of two, for some rows of a warp or all; scores that are NaN or infinite."""

import pytest
import torch

from fast_ulysses_b200.ops import attention, gemm

pytestmark = pytest.mark.gpu


def run(q, k, v):
    o, lse = attention.fmha_fwd(q, k, v)
    gemm.check_errors()
    o_ref, lse_ref = attention.attention_reference(q, k, v)
    # P and o are rounded to bf16: 2^-9 each
    assert ((o.float() - o_ref).norm() / o_ref.norm()).item() < 1e-2
    # the dominant scores are sums of 128 products in fp32, in another order (|q| |k| bounds the terms)
    terms = q.float().norm(dim=-1).max() * k.float().norm(dim=-1).max() / 128 ** 0.5
    bound = 1e-3 + 2.0 ** -20 * lse_ref.abs() + 128 * 2.0 ** -24 * terms
    assert torch.all((lse - lse_ref).abs() <= bound), (lse - lse_ref).abs().max().item()


@pytest.fixture(autouse=True)
def fp32_oracle():
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    yield
    torch.backends.cuda.matmul.allow_tf32 = before


@pytest.mark.parametrize("where", [0, 40, 70, 100, 127, 128 + 5, 128 + 120, 300])
@pytest.mark.parametrize("size", [3.0, 12.0, 60.0])
@pytest.mark.parametrize("rows", ["all", "some"])
def test_reference_moves_up(where, size, rows):
    torch.manual_seed(where)
    q = torch.randn(1, 256, 2, 128, device="cuda").bfloat16()
    k = torch.randn(1, 333, 2, 128, device="cuda").bfloat16()
    v = torch.randn(1, 333, 2, 128, device="cuda").bfloat16()
    hot = q[:, 5] if rows == "some" else q.float().mean(1).bfloat16() * 16
    k[:, where] = hot * size  # one key that some, or about half, of the queries match very well
    run(q, k, v)


@pytest.mark.parametrize("level", [-40.0, -4.0, 4.0, 40.0])
def test_reference_of_the_first_step(level):
    torch.manual_seed(3)
    q = torch.randn(1, 128, 1, 128, device="cuda").abs().bfloat16()
    k = (torch.randn(1, 200, 1, 128, device="cuda") * 0.1 + level).bfloat16()  # every score far from zero, all alike
    v = torch.randn(1, 200, 1, 128, device="cuda").bfloat16()
    run(q, k, v)


def test_first_step_far_below_a_later_one():
    torch.manual_seed(4)
    q = torch.randn(1, 128, 1, 128, device="cuda").abs().bfloat16()
    k = torch.full((1, 512, 1, 128), -30.0, device="cuda").bfloat16()
    k[:, 384:] = (torch.randn(1, 128, 1, 128, device="cuda") + 30.0).bfloat16()
    v = torch.randn(1, 512, 1, 128, device="cuda").bfloat16()
    run(q, k, v)


# 256 query rows are an item; items beyond whole waves of one per SM are shared out to clusters of up to
# eight CTAs, each with a part of the 128-row kv tiles
@pytest.mark.parametrize("b,h,sq,skv", [(1, 1, 1, 129), (1, 1, 256, 256), (1, 2, 300, 384), (1, 1, 257, 500), (2, 1, 130, 640),
                                        (1, 1, 64, 1025), (1, 3, 700, 1111), (1, 1, 256, 8 * 128 + 1), (1, 1, 100, 6000),
                                        (1, 8, 1000, 1000), (1, 20, 1024, 400), (1, 37, 1000, 300), (2, 19, 1030, 1500),
                                        (1, 1, 257, 3000), (1, 3, 700, 4111), (1, 10, 1000, 3333), (1, 9, 2000, 2600), (1, 40, 1024, 2000)])
def test_kv_tiles_shared_by_a_cluster(b, h, sq, skv):
    torch.manual_seed(sq + skv)
    q = torch.randn(b, sq, h, 128, device="cuda").bfloat16()
    k = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    v = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    k[:, skv // 2:] *= 1.5  # the shares see different ranges of scores
    run(q, k, v)
    k[:, skv - 1] = q[:, sq // 2] * 20.0  # the last share moves its reference for some rows
    run(q, k, v)
    first = attention.fmha_fwd(q, k, v)
    assert all(torch.equal(x, y) for x, y in zip(first, attention.fmha_fwd(q, k, v)))


# one query tile per item, its even and odd kv tiles through either half of the kernel
@pytest.mark.parametrize("b,h,sq,skv", [(1, 1, 1, 129), (1, 2, 128, 256), (1, 3, 257, 300), (2, 1, 130, 384), (1, 5, 1000, 640),
                                        (2, 5, 1000, 1000), (1, 20, 1000, 1025), (1, 148, 128, 200), (1, 149, 128, 500)])
def test_kv_tiles_by_parity(b, h, sq, skv):
    torch.manual_seed(sq * 5 + skv)
    q = torch.randn(b, sq, h, 128, device="cuda").bfloat16()
    k = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    v = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    run(q, k, v)
    first = attention.fmha_fwd(q, k, v)
    assert all(torch.equal(x, y) for x, y in zip(first, attention.fmha_fwd(q, k, v)))
    for at, size in ((0, 20.0), (min(130, skv - 1), 40.0), (skv - 1, 90.0)):  # either half moves its reference, and far
        k[:, at] = q[:, sq // 2] * size
        run(q, k, v)


# backward: 128 kv rows are an item, and the 128-row query blocks are what a cluster shares
@pytest.mark.parametrize("b,h,sq,skv", [(1, 1, 256, 40), (1, 1, 1025, 64), (1, 1, 640, 129), (1, 2, 2000, 300), (2, 3, 1111, 700),
                                        (1, 1, 8 * 128 + 1, 128), (1, 8, 1500, 1000), (1, 20, 1024, 1024), (1, 37, 1500, 600)])
def test_query_blocks_shared_by_a_cluster(b, h, sq, skv):
    torch.manual_seed(sq + skv)
    q = torch.randn(b, sq, h, 128, device="cuda").bfloat16()
    k = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    v = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    o, lse = attention.fmha_fwd(q, k, v)
    d_o = torch.randn_like(o)
    grads = attention.fmha_bwd(q, k, v, o, lse, d_o)
    again = attention.fmha_bwd(q, k, v, o, lse, d_o)
    whole = attention.fmha_bwd(q, k, v, o, lse, d_o, ctas=148)  # an explicit grid shares nothing
    gemm.check_errors()
    assert torch.equal(grads[1], again[1]) and torch.equal(grads[2], again[2])
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref, _ = attention.attention_reference(qr, kr, vr)
    o_ref.backward(d_o.float())
    for name, got, want, plain in zip("qkv", grads, (qr.grad, kr.grad, vr.grad), whole):
        # P, dS and the gradient are rounded to bf16: 2^-9 each
        assert ((got.float() - want).norm() / want.norm().clamp_min(1e-6)).item() < 1e-2, name
        # the same terms, summed in fp32 in another order and rounded once: one step of bf16 apart at most
        # where the sum is not cancelled, so 2^-9 in the norm with room to spare
        assert ((got.float() - plain.float()).norm() / plain.float().norm().clamp_min(1e-6)).item() < 2.0 ** -9, name


# two query tiles per item, clusters that share the kv tiles, and one query tile with its kv tiles by parity
FORMS = [(1, 1, 256, 700, 148), (1, 10, 4000, 1500, 0), (1, 2, 300, 700, 0)]


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
@pytest.mark.parametrize("where", [0, 1, 2, 5, 96, 97, 127, 128, 136, 300, -60, -59, -2, -1])  # from -60 on: the ragged last tile
def test_nan_in_a_key_reaches_every_row(b, h, sq, skv, ctas, where):
    torch.manual_seed(where + 60)
    q, k, v = (torch.randn(b, s, h, 128, device="cuda").bfloat16() for s in (sq, skv, skv))
    k[:, where, 0, 7] = float("nan")
    o, lse = attention.fmha_fwd(q, k, v, ctas=ctas)
    gemm.check_errors()
    assert o[:, :, 0].isnan().all() and lse[:, 0].isnan().all()
    assert not o[:, :, 1:].isnan().any() and not lse[:, 1:].isnan().any()  # the other heads


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
def test_nan_in_a_query_stays_in_its_row(b, h, sq, skv, ctas):
    torch.manual_seed(5)
    q, k, v = (torch.randn(b, s, h, 128, device="cuda").bfloat16() for s in (sq, skv, skv))
    q[:, 77, 0, 3] = float("nan")
    o, lse = attention.fmha_fwd(q, k, v, ctas=ctas)
    gemm.check_errors()
    bad = torch.zeros(b, sq, h, dtype=torch.bool, device="cuda")
    bad[:, 77, 0] = True
    assert torch.equal(o.isnan().any(-1), bad) and torch.equal(o.isnan().all(-1), bad)
    assert torch.equal(lse.isnan(), bad.transpose(1, 2))


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
def test_a_weight_that_underflows_is_zero(b, h, sq, skv, ctas):
    """Half the keys of every tile score hundreds of powers of two below the rest, and their values are the
    largest there are (2^127): a weight of exactly zero keeps them out."""
    torch.manual_seed(6)
    q = torch.randn(b, sq, h, 128, device="cuda").abs().bfloat16()
    k, v = (torch.randn(b, skv, h, 128, device="cuda").bfloat16() for _ in range(2))
    hidden = torch.arange(skv, device="cuda") % 16 < 8
    k[:, hidden] = -50.0
    v[:, hidden] = 2.0 ** 127
    o, lse = attention.fmha_fwd(q, k, v, ctas=ctas)
    gemm.check_errors()
    o_ref, lse_ref = attention.attention_reference(q, k[:, ~hidden], v[:, ~hidden])
    assert ((o.float() - o_ref).norm() / o_ref.norm()).item() < 1e-2  # P and o are rounded to bf16: 2^-9 each
    assert ((lse - lse_ref).abs().max()).item() < 1e-3


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
@pytest.mark.parametrize("first,last", [(0, 1), (0, 128), (128, 256), (0, 256), (256, 512), (100, 400), (0, 690), (512, 700)])
def test_steps_whose_scores_are_all_minus_infinity(b, h, sq, skv, ctas, first, last):
    """Keys ruled out by a score of -inf, a whole kv step or several of them, wherever a form begins: its first
    step, the first of the odd steps, the first of a share. Only every other query rules them out."""
    torch.manual_seed(first + last)
    q, k, v = (torch.randn(b, s, h, 128, device="cuda").bfloat16() for s in (sq, skv, skv))
    q[..., 0] = 1.0
    q[:, 1::2, :, 0] = 0.0
    keep = torch.ones(skv, dtype=torch.bool, device="cuda")
    keep[first:last] = False
    k[:, ~keep, :, 0] = -torch.inf
    o, lse = attention.fmha_fwd(q, k, v, ctas=ctas)
    gemm.check_errors()
    o_ref, lse_ref = attention.attention_reference(q[:, ::2], k[:, keep], v[:, keep])
    assert ((o[:, ::2].float() - o_ref).norm() / o_ref.norm()).item() < 1e-2  # P and o are rounded to bf16: 2^-9 each
    assert ((lse[..., ::2] - lse_ref).abs().max()).item() < 1e-3
    assert o[:, 1::2].isnan().all()  # 0 x -inf


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS + [(1, 2, 200, 1, 0), (1, 2, 200, 128, 0)])
@pytest.mark.parametrize("where", [0, 1, 50, 127, 128, 200, -1])
def test_a_weight_of_one_is_exact(b, h, sq, skv, ctas, where):
    """One key outweighs all others by 2^28: the result is its value, bit for bit, because a reference taken from it
    makes its weight 1 in bf16."""
    torch.manual_seed(where + 1)
    q, k = torch.zeros(b, sq, h, 128, device="cuda"), torch.zeros(b, skv, h, 128, device="cuda")
    v = torch.randn(b, skv, h, 128, device="cuda").bfloat16()
    where = min(where, skv - 1)
    q[..., 0], k[:, where, :, 0] = 7.0, 31.375  # x log2(e) / sqrt(128): 28.006, whose power of two lies between two bf16 numbers
    o, lse = attention.fmha_fwd(q.bfloat16(), k.bfloat16(), v, ctas=ctas)
    gemm.check_errors()
    assert torch.equal(o, v[:, where].unsqueeze(1).expand_as(o))


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
@pytest.mark.parametrize("score", [1.0078125, 1.9765625, 3.9375])  # x 8 log2(e) / sqrt(128): their powers of two, too
def test_equal_scores_average_the_values(b, h, sq, skv, ctas, score):
    """Every weight is the same and rounds the same way: only a weight that bf16 holds leaves no error behind."""
    torch.manual_seed(7)
    q, k = torch.zeros(b, sq, h, 128, device="cuda"), torch.zeros(b, skv, h, 128, device="cuda")
    v = (torch.randn(b, skv, h, 128, device="cuda") + 2.0).bfloat16()
    q[..., 0], k[..., 0] = 8.0, score
    o, _ = attention.fmha_fwd(q.bfloat16(), k.bfloat16(), v, ctas=ctas)
    gemm.check_errors()
    mean = v.double().mean(1, keepdim=True).expand_as(o)
    # one rounding to bf16 (half a unit in the last of 8 bits) and fp32 sums of a thousand terms
    assert torch.all((o.double() - mean).abs() <= mean.abs() * 2.0 ** -8 * 1.002 + 1e-5)


@pytest.mark.parametrize("b,h,sq,skv,ctas", FORMS)
@pytest.mark.parametrize("scale", [-0.1, 0.0, 0.7])
def test_any_scale(b, h, sq, skv, ctas, scale):
    """The reference is a maximum of scores before they are scaled: with a negative scale, the smallest exponent."""
    torch.manual_seed(8)
    q, k, v = (torch.randn(b, s, h, 128, device="cuda").bfloat16() for s in (sq, skv, skv))
    o, lse = attention.fmha_fwd(q, k, v, scale=scale, ctas=ctas)
    gemm.check_errors()
    o_ref, lse_ref = attention.attention_reference(q, k, v, scale=scale)
    assert ((o.float() - o_ref).norm() / o_ref.norm()).item() < 1e-2  # P and o are rounded to bf16: 2^-9 each
    assert ((lse - lse_ref).abs().max()).item() < 1e-3


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("scale", [-0.1, 0.0])
def test_gradients_at_any_scale(scale, deterministic):
    torch.manual_seed(9)
    q, k, v = (torch.randn(1, s, 2, 128, device="cuda").bfloat16() for s in (200, 300, 300))
    o, lse = attention.fmha_fwd(q, k, v, scale=scale)
    d_o = torch.randn_like(o)
    grads = attention.fmha_bwd(q, k, v, o, lse, d_o, scale=scale, deterministic=deterministic)
    gemm.check_errors()
    ref = [t.float().requires_grad_() for t in (q, k, v)]
    attention.attention_reference(*ref, scale=scale)[0].backward(d_o.float())
    for got, want in zip(grads, ref):
        # P, dS and the gradient are rounded to bf16: 2^-9 each
        assert ((got.float() - want.grad).norm() / want.grad.norm().clamp_min(1e-6)).item() < 1e-2
