"""A kernel that its caller limits to some CTAs leaves the other SMs to other streams, also when a kernel is queued behind it."""

import pytest
import torch

from fast_ulysses_b200.ops import attention, gemm

pytestmark = pytest.mark.gpu

CTAS = 74  # half of the SMs


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def _limited(kind):
    """A call of most of a millisecond on CTAS SMs."""
    if kind == "forward":
        q = _rand(1, 16384, 3, 128)
        out = torch.empty_like(q)
        return lambda: attention.fmha_fwd(q, q, q, out=out, ctas=CTAS)
    if kind == "backward":  # its last kernel, with CTAs for the whole device, comes behind the limited one
        q = _rand(1, 8192, 4, 128)
        o, lse = attention.fmha_fwd(q, q, q)
        grads = [torch.empty_like(q) for _ in range(3)]
        return lambda: attention.fmha_bwd(q, q, q, o, lse, q, out=grads, ctas=CTAS)
    a, b = _rand(8192, 8192), _rand(4096, 8192)
    out = torch.empty(8192, 4096, device="cuda", dtype=torch.bfloat16)
    return lambda: gemm.gemm_bf16(a, b, out=out, ctas=CTAS, pair=kind == "pairs")


# behind it another one with a limit, which would take just the other half; or one without
@pytest.mark.parametrize("behind", [CTAS, 0])
@pytest.mark.parametrize("kind", ["pairs", "tiles", "forward", "backward"])
def test_other_streams_find_the_rest_free(kind, behind):
    first = _limited(kind)
    a, b, out = _rand(4096, 512), _rand(4096, 512), _rand(4096, 4096)
    x, w, y = _rand(1280, 512), _rand(768, 512), _rand(1280, 768)  # 60 CTAs
    side, share = torch.cuda.Stream(), []

    def step():
        start, done, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        start.record()
        first()
        gemm.gemm_bf16(a, b, out=out, ctas=behind)
        end.record()
        with torch.cuda.stream(side):
            torch.cuda._sleep(100000)  # until the two above are on the device
            gemm.gemm_bf16(x, w, out=y, pair=False)
            done.record()
        torch.cuda.synchronize()
        share.append(start.elapsed_time(done) / start.elapsed_time(end))

    for _ in range(4):
        step()
    gemm.check_errors()
    # 0.1 ms of 0.7 or more; behind the kernel that is queued, all of it
    assert min(share[1:]) < 0.6, share
