"""Kernels that are set up while the one before them still runs: each reads what that one wrote, one behind the other with no
host in between, and replayed. The oracle is the same program in a process where every launch waits for the one before
(CUDA_LAUNCH_BLOCKING); that its results are right is what the other tests say."""

import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

if __name__ == "__main__":  # the oracle's process
    sys.path.insert(0, str(Path(__file__).resolve().parents[1]))

import fast_ulysses_b200 as fu
from fast_ulysses_b200.models.dit import DiTBlock
from fast_ulysses_b200.ops import attention, fp8, gemm, norm

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


def _forward(group, m, heads, ffn):
    """LayerNorm, both GEMMs, attention and a projection in a ring, each reading what the kernel right before it wrote."""
    hidden = heads * 128
    x0, w1, b1 = _rand(1, m, hidden), _rand(ffn, hidden, scale=0.05), _rand(ffn)
    w2, b2, w3, b3 = _rand(hidden, ffn, scale=0.05), _rand(hidden), _rand(hidden, hidden, scale=0.05), _rand(hidden)

    def step():
        x = x0
        for _ in range(3):
            y = gemm.feed_forward(norm.layer_norm(x, 1e-6), w1, b1, w2, b2, residual=x)
            q = norm.layer_norm(y, 1e-6).view(1, m, heads, 128)
            x = gemm.linear(attention.attention(q, q, q).view(1, m, hidden), w3, b3, residual=y)
        return [x]

    return step


def _exchange(group, m, heads, ffn):
    """Exchanges between two buffers and the fp8 form, behind a LayerNorm and one another: each writes what the next reads, and
    over what the one before has read."""
    hidden = heads * 128
    x0 = _rand(1, m, heads, 128)
    a, b = (group.empty_output(x0) for _ in range(2))

    def step():
        x = x0
        for _ in range(3):
            y = norm.layer_norm(x.view(1, m, hidden), 1e-6).view(1, m, heads, 128)
            group.all_to_all_4d(y, out=a)
            group.all_to_all_4d(a, mode=1, out=b)
            group.all_to_all_4d(b, out=a)
            x = fp8.all_to_all_4d_fp8(group, a)
        return [x, group.all_to_all_4d(x)]

    return step


def _sums(group, m, heads, ffn):
    """Two linear layers with biases, forward and backward: column sums behind the GEMM whose result they read."""
    hidden = heads * 128
    leaves = [_rand(m, hidden), _rand(ffn, hidden, scale=0.05), _rand(ffn), _rand(hidden, ffn, scale=0.05), _rand(hidden)]
    dy = _rand(m, hidden)
    for t in leaves:
        t.requires_grad_()

    def step():
        x, w1, b1, w2, b2 = leaves
        y = gemm.linear(norm.layer_norm(gemm.linear(x, w1, b1), 1e-6), w2, b2)
        return [y.detach(), *torch.autograd.grad(y, leaves, dy)]

    return step


def _block(group, m, heads, ffn):
    """A training step of a whole block: projection, gradient pull, attention's and LayerNorm's backward among its kernels."""
    block = DiTBlock(group, heads * 128, heads, ffn, grid=(2, m // 20, 10))
    x, dy = _rand(1, m, heads * 128).requires_grad_(), _rand(1, m, heads * 128)
    leaves = [x, *block.parameters()]

    def step():
        y = block(x)
        return [y.detach(), *torch.autograd.grad(y, leaves, dy)]

    return step


PROGRAMS = {"forward": _forward, "exchange": _exchange, "sums": _sums, "block": _block}
# one tile and several, single CTAs and pairs, attention of whole and of single query tiles; LayerNorm's rows of one, two, four and
# eight warps, and a matrix whose backward walks through them
SIZES = [(20, 1, 64), (140, 2, 520), (1100, 5, 2048), (4100, 12, 1536), (4000, 25, 512), (20, 41, 64)]


def _prepared(name, size, group):
    torch.manual_seed(size[0])
    return PROGRAMS[name](group, *size)


@pytest.fixture(scope="module")
def serial(tmp_path_factory):
    path = tmp_path_factory.mktemp("serial") / "want.pt"
    subprocess.run([sys.executable, __file__, str(path)], check=True, timeout=300, env=dict(os.environ, CUDA_LAUNCH_BLOCKING="1"))
    return torch.load(path)


@pytest.fixture(scope="module")
def group():
    g = fu.UlyssesGroup(device="cuda")
    yield g
    g.check()
    g.destroy()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("name", PROGRAMS)
def test_a_chain_behind_itself_and_replayed(serial, group, name, size):
    want = [t.cuda() for t in serial[name, size]]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()  # one that may be captured, with all of the autograd graph on it
    with torch.cuda.stream(stream):
        step = _prepared(name, size, group)
        step()
        torch.cuda.synchronize()
        many = [step() for _ in range(4)]  # nothing waits until all are queued
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = step()
        for _ in range(3):
            for t in out:
                t.zero_()
            graph.replay()
            many.append([t.clone() for t in out])
    torch.cuda.synchronize()
    for got in many:
        for a, b in zip(got, want):
            if name != "block":
                assert torch.equal(a, b)
            else:  # dQ and d(gamma) are summed by atomics in any order, then rounded to bf16: half a unit, 2^-9
                assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 4e-3
    gemm.check_errors()


if __name__ == "__main__":
    assert os.environ["CUDA_LAUNCH_BLOCKING"] == "1"
    alone = fu.UlyssesGroup(device="cuda")
    torch.save({(name, size): [t.detach().cpu() for t in _prepared(name, size, alone)()] for name in PROGRAMS for size in SIZES}, sys.argv[1])
    alone.destroy()
