"""The GEMM cores at the edges of their schedules: one accumulator block of a tile outside the result, a
last wave split into blocks, K shorter than the ring, as long as it, and one K-block more; both operand
layouts; every epilogue on ragged columns. Oracle: the same contraction in fp32."""

import pytest
import torch

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
# clusters of two or four pairs along K; with and without a launch before it, ragged in every direction
@pytest.mark.parametrize("act", [0, 1, 3])
@pytest.mark.parametrize("m,n,k", [(1000, 5120, 5120), (512, 5120, 6016), (2000, 5128, 2568), (1800, 5000, 4104), (257, 10000, 4096),
                                   (4100, 4096, 1544), (2048, 5120, 5120)])
def test_rest_shared_by_clusters_of_pairs(act, m, n, k):
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(n, k, device="cuda") * 0.02).bfloat16()
    bias, res, aux = torch.randn(n, device="cuda"), torch.randn(m, n, device="cuda").bfloat16(), torch.randn(m, n, device="cuda").bfloat16()
    pre = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    kw = dict(bias=bias, residual=res, act=act, aux=aux if act == 3 else None)
    got = gemm.gemm_bf16(a, b, store_pre=pre, **kw)
    again = gemm.gemm_bf16(a, b, **kw)
    whole = gemm.gemm_bf16(a, b, pair=True, **kw)
    turned = gemm.gemm_bf16(a.t().contiguous(), b.t().contiguous(), a_km=True, b_kn=True, **kw) if m % 8 == 0 else got
    gemm.check_errors()
    assert torch.equal(got, again) and torch.equal(got, turned)
    # the same products summed in fp32 in another order, then rounded to bf16 once
    assert rel_err(got, whole.float()) < 1e-3
    assert rel_err(pre, a.float() @ b.float().t() + bias) < 4e-3
