"""Kernels that are set up while the one before them still runs: each reads what that one wrote, run behind it and replayed."""

import pytest
import torch

from fast_ulysses_b200.ops import attention, gemm, norm

pytestmark = pytest.mark.gpu


def _chain(x, w1, b1, w2, b2, heads):
    """Every kernel reads what the kernel right before it wrote, and writes where an earlier one has read."""
    m, hidden = x.shape[1:]
    for _ in range(3):
        y = norm.layer_norm(x, 1e-6)
        y = gemm.feed_forward(y, w1, b1, w2, b2, residual=x)
        q = y.view(1, m, heads, 128)
        x = (x + attention.attention(q, q, q).reshape(1, m, hidden)) * 0.5
    return x


# one tile and several, single CTAs and pairs, a forward pass of whole and of single query tiles
@pytest.mark.parametrize("m,heads,ffn", [(1, 1, 64), (129, 2, 520), (1100, 5, 2048), (4100, 12, 1536)])
def test_a_chain_behind_itself_and_replayed(m, heads, ffn):
    torch.manual_seed(m)
    hidden = heads * 128
    x = torch.randn(1, m, hidden, device="cuda").bfloat16()
    w1, w2 = ((torch.randn(*s, device="cuda") * 0.05).bfloat16() for s in ((ffn, hidden), (hidden, ffn)))
    b1, b2 = torch.randn(ffn, device="cuda").bfloat16(), torch.randn(hidden, device="cuda").bfloat16()
    with torch.no_grad():
        want = _chain(x, w1, b1, w2, b2, heads)
        torch.cuda.synchronize()
        for _ in range(5):  # nothing but these kernels between one chain and the next
            got = _chain(x, w1, b1, w2, b2, heads)
            assert torch.equal(got, want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _chain(x, w1, b1, w2, b2, heads)
        for _ in range(3):
            out.zero_()
            graph.replay()
            assert torch.equal(out, want)
    gemm.check_errors()
