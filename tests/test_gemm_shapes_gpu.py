"""The GEMM cores at the edges of their schedules: one accumulator block of a tile outside the result, a
last wave split into blocks, K shorter than the ring, as long as it, and one K-block more; both operand
layouts; every epilogue on ragged columns. Oracle: the same contraction in fp32."""

import pytest
import torch

from _graph import kernel_names
from fast_ulysses_b200.ops import gemm

pytestmark = pytest.mark.gpu


def rel_err(got, want):
    return ((got.float() - want).norm() / want.norm().clamp_min(1e-12)).item()


# 148 SMs hold 74 pairs: 75 tiles leave one tile of two blocks, 37 + 74 exactly half a wave of blocks
@pytest.mark.parametrize("m,n", [(256, 512), (257, 512), (512, 256), (512, 257), (300, 300), (256 * 75, 512), (512 * 37, 768),
                                 (128, 128 * 149), (1, 8)])
@pytest.mark.parametrize("k", [8, 64, 256, 264, 576])
def test_schedules(m, n, k):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16()
    pitch = (n + 7) // 8 * 8
    want = a.float() @ b.float().t()
    out = {}
    for pair in (True, False, None):
        buf = torch.full((m, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
        out[pair] = gemm.gemm_bf16(a, b, pair=pair, out=buf[:, :n])
        gemm.check_errors()
        assert (buf[:, n:] == 7.0).all()
    # bf16 rounding of the result: 2^-9 relative, a little more for the fp32 sums
    assert rel_err(out[True], want) < 4e-3
    assert torch.equal(out[True], out[False]) and torch.equal(out[True], out[None])


@pytest.mark.parametrize("pair", [True, False])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
@pytest.mark.parametrize("m,n,k", [(257, 520, 72), (129, 136, 320)])
def test_epilogues_on_ragged_tiles(pair, act, m, n, k):
    torch.manual_seed(act)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(n, k, device="cuda") * 0.2).bfloat16()
    bias, res, aux = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda").bfloat16(), torch.randn(m, n, device="cuda").bfloat16()
    pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    got = gemm.gemm_bf16(a, b, bias=bias, residual=res, act=act, aux=aux if act == 3 else None, store_pre=pre, pair=pair)
    gemm.check_errors()
    y = a.double() @ b.double().t() + bias.double()
    assert rel_err(pre, y.float()) < 4e-3
    if act == 1:
        y = torch.nn.functional.gelu(y, approximate="tanh")
    elif act == 2:
        y = torch.nn.functional.gelu(y)
    elif act == 3:
        x = aux.double().requires_grad_()
        torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
        y = y * x.grad
    assert rel_err(got, (y + res.double()).float()) < 4e-3


# few tiles and a long K: two, four or eight CTAs share the K-blocks of a tile, the last with fewer
@pytest.mark.parametrize("act", [0, 1, 3])
@pytest.mark.parametrize("m,n,k", [(1, 8, 8192), (128, 128, 4104), (129, 264, 3000), (64, 1000, 8000), (300, 520, 5000),
                                   (500, 1600, 4096), (700, 1416, 4160), (1000, 1024, 6000)])
def test_k_shared_by_a_cluster(act, m, n, k):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(n, k, device="cuda") * 0.02).bfloat16()
    bias, res, aux = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda").bfloat16(), torch.randn(m, n, device="cuda").bfloat16()
    pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    kw = dict(bias=bias, residual=res, act=act, aux=aux if act == 3 else None)
    got = gemm.gemm_bf16(a, b, store_pre=pre, **kw)
    again = gemm.gemm_bf16(a, b, **kw)
    whole = gemm.gemm_bf16(a, b, pair=False, **kw)
    turned = gemm.gemm_bf16(a.t().contiguous(), b.t().contiguous(), a_km=True, b_kn=True, **kw) if m % 8 == 0 else got
    gemm.check_errors()
    assert torch.equal(got, again) and torch.equal(got, turned)
    y = a.double() @ b.double().t() + bias.double()
    assert rel_err(pre, y.float()) < 4e-3
    # the same products summed in fp32 in another order, then rounded to bf16 once: equal but for a few
    # results that lie at the edge between two bf16 numbers
    assert rel_err(got, whole.float()) < 1e-3
    if act == 1:
        y = torch.nn.functional.gelu(y, approximate="tanh")
    elif act == 3:
        x = aux.double().requires_grad_()
        torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
        y = y * x.grad
    assert rel_err(got, (y + res.double()).float()) < 4e-3


# more 256 x 256 blocks than whole waves of pairs: the rest, some of it outside the result, is shared by
# clusters of two or four pairs along K; with and without a launch before it, ragged in every direction. (With B
# the other way round narrower blocks are mostly preferred.)
@pytest.mark.parametrize("act", [0, 1, 3])
@pytest.mark.parametrize("m,n,k", [(1000, 5120, 5120), (2000, 5120, 5120), (798, 5400, 3208), (4100, 1536, 4096), (1800, 5000, 4104)])
def test_rest_shared_by_clusters_of_pairs(act, m, n, k):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(k, n, device="cuda") * 0.02).bfloat16()
    bias, res, aux = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda").bfloat16(), torch.randn(m, n, device="cuda").bfloat16()
    pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    kw = dict(bias=bias, residual=res, act=act, aux=aux if act == 3 else None, b_kn=True)
    got = gemm.gemm_bf16(a, b, store_pre=pre, **kw)
    again = gemm.gemm_bf16(a, b, **kw)
    whole = gemm.gemm_bf16(a, b, pair=True, **kw)
    gemm.check_errors()
    assert torch.equal(got, again)
    # the same products summed in fp32 in another order, then rounded to bf16 once
    assert rel_err(got, whole.float()) < 1e-3
    assert rel_err(pre, a.float() @ b.float() + bias) < 4e-3


# blocks of 160, 192, 224 and 256 columns, one to a pair or two beside or under each other: one wave, a wave
# and a bit, the last block inside and beyond the edge of the result
@pytest.mark.parametrize("act", [0, 3])
@pytest.mark.parametrize("m,n,k", [(388, 4744, 2696), (265, 6304, 2432), (258, 7208, 3088), (517, 5392, 2352), (1060, 2072, 984),
                                   (663, 3856, 1104), (1033, 5440, 1720), (802, 2704, 1112), (798, 2912, 1152), (774, 7152, 2904),
                                   (512, 5120, 704), (3491, 2592, 3000)])
def test_narrow_and_single_blocks(act, m, n, k):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    bias, res, aux = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda").bfloat16(), torch.randn(m, n, device="cuda").bfloat16()
    kw = dict(bias=bias, residual=res, act=act, aux=aux if act == 3 else None)
    for layout in ({}, {"b_kn": True}):
        other = b.t().contiguous() if layout else b
        buf = torch.full((m, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        got = gemm.gemm_bf16(a, other, out=buf[:, :n], bias=bias, **layout)
        assert (buf[:, n:] == 7.0).all()
        assert rel_err(got, a.float() @ b.float().t() + bias) < 4e-3
        # the same products summed in fp32, perhaps in another order, then rounded to bf16 once
        whole = gemm.gemm_bf16(a, other, pair=True, **kw, **layout)
        assert rel_err(gemm.gemm_bf16(a, other, **kw, **layout), whole.float()) < 1e-3
    gemm.check_errors()


# few tiles of two blocks, all of which would be run block by block: the kernel for that, or small tiles, does
@pytest.mark.parametrize("m,n,k,act,b_kn", [(1024, 2432, 512, 0, False), (1024, 2432, 512, 2, False),
                                            (143, 10928, 12416, 0, True), (1216, 2528, 8112, 0, True), (4105, 288, 9032, 2, False)])
def test_halves_of_tiles_are_single_blocks(m, n, k, act, b_kn):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(*((k, n) if b_kn else (n, k)), device="cuda") * 0.05).bfloat16()
    kw = dict(act=act, b_kn=b_kn)
    names = kernel_names(lambda: gemm.gemm_bf16(a, b, **kw))
    assert len(names) == 1 and any(kernel in names[0] for kernel in ("gemm_wide_kernelILi1ELi1E", "gemm_small_kernel", "gemm_split_kernel")), names
    # the same products summed in fp32, perhaps in another order, then rounded to bf16 once
    assert rel_err(gemm.gemm_bf16(a, b, **kw), gemm.gemm_bf16(a, b, pair=True, **kw).float()) < 1e-3
    gemm.check_errors()


# single blocks on pairs, whose operands have a producer each: many items to a pair, K one block short of the ring of six, as long,
# longer by one, twice round and more with a part; then one item to a pair or two, of 160 to 256 columns. Both kinds of B.
@pytest.mark.parametrize("m,n,k,b_kn,ctas", [(905, 936, 320, True, 4), (1348, 160, 384, False, 4), (928, 920, 384, True, 4), (1286, 160, 448, False, 4),
                                             (922, 904, 448, True, 4), (1441, 400, 768, False, 4), (641, 1160, 768, True, 4),
                                             (641, 528, 1032, False, 4), (1159, 656, 1032, True, 4), (388, 4744, 2696, False, 0),
                                             (265, 6304, 2432, False, 0), (258, 7208, 3088, True, 0), (802, 2704, 1112, False, 0)])
def test_single_blocks_with_a_producer_for_each_operand(m, n, k, b_kn, ctas):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b = torch.randn(m, k, device="cuda", generator=gen).bfloat16(), torch.randn(n, k, device="cuda", generator=gen).bfloat16()
    other = b.t().contiguous() if b_kn else b
    names = kernel_names(lambda: gemm.gemm_bf16(a, other, b_kn=b_kn, ctas=ctas))
    assert len(names) == 1 and "gemm_wide_kernelILi1ELi1E" in names[0], names
    got = gemm.gemm_bf16(a, other, b_kn=b_kn, ctas=ctas)
    gemm.check_errors()
    assert rel_err(got, a.float() @ b.float().t()) < 4e-3  # bf16 rounding of the result, as above
    assert torch.equal(got, gemm.gemm_bf16(a, b, pair=False))


# small tiles with the erf GELU: one K-block more than 16 is no reason for another kernel (pairs took a quarter longer there)
@pytest.mark.parametrize("m,n", [(1914, 7104), (1086, 4224)])
@pytest.mark.parametrize("k", [1024, 1040, 1088])
def test_shape_around_sixteen_k_blocks(m, n, k):
    torch.manual_seed(k)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    names = kernel_names(lambda: gemm.gemm_bf16(a, b, act=2))
    assert len(names) == 1 and "gemm_small_kernel" in names[0], names
    gemm.check_errors()


# a hidden layer whose rows are an odd multiple of 16 bytes is kept with a wider pitch; one that is not, as it is
@pytest.mark.parametrize("m,hidden,ffn", [(1, 8, 8), (130, 72, 264), (300, 128, 256), (257, 264, 1032)])
def test_feed_forward_with_a_padded_hidden_layer(m, hidden, ffn):
    torch.manual_seed(m)
    x = torch.randn(m, hidden, device="cuda").bfloat16().requires_grad_()
    w1 = (torch.randn(ffn, hidden, device="cuda") * 0.1).bfloat16().requires_grad_()
    w2 = (torch.randn(hidden, ffn, device="cuda") * 0.1).bfloat16().requires_grad_()
    b1 = torch.randn(ffn, device="cuda").bfloat16().requires_grad_()
    b2 = torch.randn(hidden, device="cuda").bfloat16().requires_grad_()
    gy = torch.randn(m, hidden, device="cuda").bfloat16()
    with torch.no_grad():
        plain = gemm.feed_forward(x, w1, b1, w2, b2)
    y = gemm.feed_forward(x, w1, b1, w2, b2)
    y.backward(gy)
    gemm.check_errors()
    assert torch.equal(y, plain) and y.is_contiguous()
    ref = [t.detach().float().requires_grad_() for t in (x, w1, b1, w2, b2)]
    h = torch.nn.functional.gelu(ref[0] @ ref[1].t() + ref[2], approximate="tanh")
    (h @ ref[3].t() + ref[4]).backward(gy.float())
    # the hidden layer and its gradient are rounded to bf16 on the way, and the results: 2^-9 each
    for got, want in zip((x, w1, b1, w2, b2), ref):
        assert rel_err(got.grad, want.grad) < 1e-2


# K one block short of the ring of six, as long as it, one more, and twice round; a CTA's second tile begins where the first left the ring
@pytest.mark.parametrize("k", [320, 384, 448, 768, 840])
@pytest.mark.parametrize("a_km,b_kn", [(False, False), (False, True), (True, True)])
def test_small_tiles_around_the_ring(k, a_km, b_kn):
    m, n = 128 * 150, 136
    gen = torch.Generator(device="cuda").manual_seed(k)
    a, b = torch.randn(m, k, device="cuda", generator=gen).bfloat16(), torch.randn(n, k, device="cuda", generator=gen).bfloat16()
    got = gemm.gemm_bf16(a.t().contiguous() if a_km else a, b.t().contiguous() if b_kn else b, a_km=a_km, b_kn=b_kn, pair=False)
    gemm.check_errors()
    assert rel_err(got, a.float() @ b.float().t()) < 4e-3  # bf16 rounding of the result, as above
    assert torch.equal(got, gemm.gemm_bf16(a, b, pair=True))


# a tile's columns are shared by two epilogue warps of 64: the last tile ends inside the first one's, with it, inside the second one's
@pytest.mark.parametrize("act", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [8, 56, 64, 72, 120, 128, 184, 200])
def test_small_tiles_end_in_either_half(n, act):
    gen = torch.Generator(device="cuda").manual_seed(n)
    m, k = 150, 136
    a, b = torch.randn(m, k, device="cuda", generator=gen).bfloat16(), torch.randn(n, k, device="cuda", generator=gen).bfloat16()
    bias = torch.randn(n, device="cuda", generator=gen)
    res, aux = (torch.randn(m, n, device="cuda", generator=gen).bfloat16() for _ in range(2))
    pitch, kw = n + 24, {}
    if act == 3:
        kw["aux"] = torch.empty(m, pitch, device="cuda", dtype=torch.bfloat16)[:, :n].copy_(aux)
    buf, pre = (torch.full((m, pitch), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    residual = torch.empty(m, pitch, device="cuda", dtype=torch.bfloat16)[:, :n].copy_(res)
    got = gemm.gemm_bf16(a, b, bias=bias, residual=residual, act=act, out=buf[:, :n], store_pre=pre[:, :n], pair=False, **kw)
    gemm.check_errors()
    assert (buf[:, n:] == 7.0).all() and (pre[:, n:] == 7.0).all()
    y = a.double() @ b.double().t() + bias.double()
    assert rel_err(pre[:, :n], y.float()) < 4e-3
    if act == 3:
        x = aux.double().requires_grad_()
        torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
        y = y * x.grad
    elif act:
        y = torch.nn.functional.gelu(y, approximate="tanh" if act == 1 else "none")
    assert rel_err(got, (y + res.double()).float()) < 4e-3  # bf16 rounding of the result, as above
