"""What this library's performance is measured on: a few named calls of its public entry points and
a generator of more from the same ranges. One GPU, a group of one rank.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs,
weights, the module, the group), ``run`` makes the call as a program would, ``work`` states the bytes
and operations the call cannot do without.
"""

from __future__ import annotations

import math

import torch

import fast_ulysses_b200 as fu
from fast_ulysses_b200.models.dit import DiTBlock
from fast_ulysses_b200.ops.attention import attention
from fast_ulysses_b200.ops.fp8 import all_to_all_4d_fp8
from fast_ulysses_b200.ops.gemm import feed_forward

HEAD_DIM = 128  # of the attention kernels and the block
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "int8": torch.int8}
ELEM = {"bf16": 2, "fp16": 2, "fp32": 4, "int8": 1}
WAN_TOKENS = 75600  # 21 x 45 x 80 latent positions of an 81-frame 720p video
MOST_EXCHANGE_BYTES = WAN_TOKENS * 40 * HEAD_DIM * 2
MOST_SCORES = WAN_TOKENS * WAN_TOKENS * 5

_the_group = None


def _group() -> fu.UlyssesGroup:
    """The one group a program builds at start-up."""
    global _the_group
    if _the_group is None:
        _the_group = fu.UlyssesGroup(device="cuda")
    return _the_group


def _exchange(name, b, s, n, d, dtype="bf16", mode=0, call="copy", packed=False):
    return {"name": name, "kind": "exchange", "b": b, "s": s, "n": n, "d": d, "dtype": dtype, "mode": mode, "call": call,
            "packed": packed}


def _attention(name, b, sq, skv, h, train):
    return {"name": name, "kind": "attention", "b": b, "sq": sq, "skv": skv, "h": h, "train": train}


def _block(name, t, gh, gw, heads, ffn, train):
    return {"name": name, "kind": "block", "t": t, "gh": gh, "gw": gw, "heads": heads, "ffn": ffn, "train": train}


def listed():
    return [
        # the smallest exchange of the size sweep: what one call costs when there is nothing to move
        _exchange("exchange_small", 1, 16, 40, 128),
        # the headline: q, k or v of one 720p attention layer, copying call
        _exchange("exchange_wan720p", 1, WAN_TOKENS, 40, 128),
        # a training step of an odd shape: fp32, 13 heads of 72, the inverse direction, forward and backward
        _exchange("exchange_ragged_train", 2, 4099, 13, 72, dtype="fp32", mode=1, call="train"),
        # q, k, v packed on the last axis, one rank's share of eight, asynchronous into an own symmetric buffer
        _exchange("exchange_async_packed", 1, 9478, 40, 384, call="async_out"),
        # block-scaled fp8 payload, one rank's share of eight
        {"name": "exchange_fp8", "kind": "fp8", "b": 1, "s": 9450, "n": 40, "mode": 0},
        # attention over a short sequence at inference: a single image, few heads per rank
        _attention("attention_short", 2, 1000, 1000, 5, False),
        # attention of one rank of eight at 720p: all tokens, five heads, inference
        _attention("attention_wan720p", 1, WAN_TOKENS, WAN_TOKENS, 5, False),
        # attention of a training step over a clip whose length is no multiple of any tile
        _attention("attention_train", 1, 8191, 8191, 10, True),
        # the feed-forward of a training step on one rank's share of eight
        {"name": "feed_forward_train", "kind": "ffn", "m": 9450, "hidden": 5120, "ffn": 13824, "train": True},
        # the block at the size of the smoke test: latency of a whole training step of a tiny model
        _block("block_tiny_train", 2, 8, 16, 2, 512, True),
        # the block at inference over a short clip
        _block("block_infer", 5, 30, 52, 40, 13824, False),
        # the block of a training step over the whole 720p video
        _block("block_wan720p_train", 21, 45, 80, 40, 13824, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("exchange", "exchange", "fp8", "attention", "attention", "ffn", "block"))
    if kind == "exchange":
        dtype = rng.choice(("bf16", "bf16", "fp16", "fp32", "int8"))
        d = rng.choice([v for v in (16, 64, 72, 80, 96, 128, 192, 384) if v * ELEM[dtype] % 16 == 0])
        b, n = rng.randint(1, 2), rng.randint(1, 40)
        call = rng.choice(("copy", "copy", "out", "async", "async_out") + (("train",) if dtype != "int8" else ()))
        packed = call != "train" and rng.random() < 0.3
        s = _log_int(rng, 16, max(16, min(WAN_TOKENS, MOST_EXCHANGE_BYTES // (b * n * d * ELEM[dtype]))))
        return {"kind": kind, "b": b, "s": s, "n": n, "d": d, "dtype": dtype, "mode": rng.randint(0, 1), "call": call,
                "packed": packed}
    if kind == "fp8":
        b, n = rng.randint(1, 2), rng.randint(1, 40)
        return {"kind": kind, "b": b, "s": _log_int(rng, 16, WAN_TOKENS // b), "n": n, "mode": rng.randint(0, 1)}
    if kind == "attention":
        b, h = rng.randint(1, 2), rng.randint(1, 40)
        sq = _log_int(rng, 64, min(WAN_TOKENS, int(math.sqrt(MOST_SCORES / (b * h)))))
        skv = sq if rng.random() < 0.7 else _log_int(rng, 64, min(WAN_TOKENS, int(MOST_SCORES / (b * h * sq))))
        return {"kind": kind, "b": b, "sq": sq, "skv": skv, "h": h, "train": rng.random() < 0.5}
    if kind == "ffn":
        hidden, ffn = 8 * rng.randint(32, 640), 8 * rng.randint(64, 1728)
        return {"kind": kind, "m": _log_int(rng, 64, WAN_TOKENS), "hidden": hidden, "ffn": ffn, "train": rng.random() < 0.5}
    gh, gw = rng.randint(6, 45), rng.randint(10, 80)
    return {"kind": "block", "t": _log_int(rng, 1, 21), "gh": gh, "gw": gw, "heads": rng.randint(2, 40),
            "ffn": 8 * rng.randint(64, 1728), "train": rng.random() < 0.5}


# ---- the state of a program before the call ------------------------------------------------------
class _Exchange:
    def __init__(self, c, gen):
        b, s, n, d, dtype = c["b"], c["s"], c["n"], c["d"], DTYPES[c["dtype"]]
        shape = (b, s, 3, n, d) if c["packed"] else (b, s, n, d)
        if dtype == torch.int8:
            x = torch.randint(-128, 128, shape, device="cuda", generator=gen, dtype=torch.int8)
        else:
            x = torch.randn(shape, device="cuda", generator=gen, dtype=dtype)
        self.x = x[:, :, 1] if c["packed"] else x  # packed: one of q, k, v inside a projection's output
        self.group, self.mode, self.call = _group(), c["mode"], c["call"]
        if self.call in ("out", "async_out"):
            self.out = self.group.empty_output(self.x, mode=self.mode)
        if self.call == "train":
            self.x.requires_grad_()
            self.dy = torch.randn(shape, device="cuda", generator=gen, dtype=dtype)

    def run(self):
        if self.call == "train":
            self.x.grad = None
            y = self.group.all_to_all_4d(self.x, mode=self.mode)
            y.backward(self.dy)
            return y, self.x.grad
        if self.call == "out":
            return self.group.all_to_all_4d(self.x, mode=self.mode, out=self.out)
        if self.call == "async_out":
            return self.group.all_to_all_4d_async(self.x, mode=self.mode, out=self.out).wait()
        if self.call == "async":
            return self.group.all_to_all_4d_async(self.x, mode=self.mode).wait()
        return self.group.all_to_all_4d(self.x, mode=self.mode)


class _Fp8:
    def __init__(self, c, gen):
        self.x = torch.randn(c["b"], c["s"], c["n"], HEAD_DIM, device="cuda", generator=gen, dtype=torch.bfloat16)
        self.group, self.mode = _group(), c["mode"]

    def run(self):
        return all_to_all_4d_fp8(self.group, self.x, mode=self.mode)


class _Attention:
    def __init__(self, c, gen):
        def t(s):
            return torch.randn(c["b"], s, c["h"], HEAD_DIM, device="cuda", generator=gen, dtype=torch.bfloat16)

        self.train = c["train"]
        # q and k of unit variance, as the per-head RMSNorm in front of the attention leaves them
        self.q, self.k, self.v = t(c["sq"]), t(c["skv"]), t(c["skv"])
        if self.train:
            self.d_o = t(c["sq"])
            for x in (self.q, self.k, self.v):
                x.requires_grad_()

    def run(self):
        if not self.train:
            return attention(self.q, self.k, self.v)
        self.q.grad = self.k.grad = self.v.grad = None
        o = attention(self.q, self.k, self.v)
        o.backward(self.d_o)
        return o, self.q.grad, self.k.grad, self.v.grad


class _FeedForward:
    def __init__(self, c, gen):
        def t(*shape, scale=1.0):
            return torch.randn(shape, device="cuda", generator=gen, dtype=torch.bfloat16).mul_(scale)

        m, hidden, ffn = c["m"], c["hidden"], c["ffn"]
        self.train = c["train"]
        self.x, self.residual = t(1, m, hidden), t(1, m, hidden)
        self.w1, self.b1 = t(ffn, hidden, scale=0.02), t(ffn, scale=0.02)
        self.w2, self.b2 = t(hidden, ffn, scale=0.02), t(hidden, scale=0.02)
        self.leaves = (self.x, self.w1, self.b1, self.w2, self.b2, self.residual)
        if self.train:
            self.dy = t(1, m, hidden)
            for p in self.leaves:
                p.requires_grad_()

    def run(self):
        if not self.train:
            return feed_forward(self.x, self.w1, self.b1, self.w2, self.b2, residual=self.residual)
        for p in self.leaves:
            p.grad = None
        y = feed_forward(self.x, self.w1, self.b1, self.w2, self.b2, residual=self.residual)
        y.backward(self.dy)
        return y, *(p.grad for p in self.leaves)


class _Block:
    def __init__(self, c, gen, seed):
        torch.manual_seed(seed)  # the module initialises its own weights
        hidden, grid = c["heads"] * HEAD_DIM, (c["t"], c["gh"], c["gw"])
        self.train = c["train"]
        self.block = DiTBlock(_group(), hidden, c["heads"], c["ffn"], grid=grid)
        with torch.no_grad():  # biases and norm weights as a trained model has them, not all zeros and ones
            for p in (self.block.b1, self.block.b2, self.block.attn.b_o):
                p.normal_(0.0, 0.02, generator=gen)
            for p in (self.block.attn.gamma_q, self.block.attn.gamma_k):
                p.uniform_(0.75, 1.25, generator=gen)
        shape = (1, grid[0] * grid[1] * grid[2], hidden)
        self.x = torch.randn(shape, device="cuda", generator=gen, dtype=torch.bfloat16)
        if self.train:
            self.dy = torch.randn(shape, device="cuda", generator=gen, dtype=torch.bfloat16)
            self.x.requires_grad_()
        self.params = list(self.block.parameters())

    def run(self):
        if not self.train:
            with torch.no_grad():
                return self.block(self.x)
        self.x.grad = None
        self.block.zero_grad(set_to_none=True)
        y = self.block(self.x)
        y.backward(self.dy)
        return y, self.x.grad, *(p.grad for p in self.params)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "exchange":
        return _Exchange(case, gen)
    if kind == "fp8":
        return _Fp8(case, gen)
    if kind == "attention":
        return _Attention(case, gen)
    if kind == "ffn":
        return _FeedForward(case, gen)
    return _Block(case, gen, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "exchange":
        n = case["b"] * case["s"] * case["n"] * case["d"] * ELEM[case["dtype"]]
        return {"bytes": (4 if case["call"] == "train" else 2) * n, "flops": 0}
    if kind == "fp8":
        return {"bytes": 2 * case["b"] * case["s"] * case["n"] * HEAD_DIM * 2, "flops": 0}
    if kind == "attention":
        b, sq, skv, h, train = (case[k] for k in ("b", "sq", "skv", "h", "train"))
        rows = 2 * sq + 2 * skv  # q, o and k, v
        if train:
            rows += 2 * sq + 2 * skv  # the gradient of o comes in, those of q, k, v go out
        return {"bytes": b * rows * h * HEAD_DIM * 2, "flops": (14 if train else 4) * b * h * sq * skv * HEAD_DIM}
    if kind == "ffn":
        m, hidden, ffn, train = (case[k] for k in ("m", "hidden", "ffn", "train"))
        values = 3 * m * hidden + 2 * hidden * ffn + hidden + ffn
        if train:
            values += 3 * m * hidden + 2 * hidden * ffn + hidden + ffn
        return {"bytes": 2 * values, "flops": (12 if train else 4) * m * hidden * ffn}
    tokens, heads, ffn, train = case["t"] * case["gh"] * case["gw"], case["heads"], case["ffn"], case["train"]
    hidden = heads * HEAD_DIM
    weights = 4 * hidden * hidden + 2 * hidden * ffn
    values = 2 * tokens * hidden + weights
    flops = 2 * tokens * weights + 4 * heads * tokens * tokens * HEAD_DIM
    if train:
        values += 2 * tokens * hidden + weights
        flops = 6 * tokens * weights + 14 * heads * tokens * tokens * HEAD_DIM
    return {"bytes": 2 * values, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("exchange", "fp8"):
        return "exact"  # bytes moved, or one defined rounding to e4m3 and back
    if kind == "block":
        return {"rel": 2e-2}  # several bf16 intermediates in a chain, forward and backward
    return {"rel": 1e-2}  # bf16 inputs and results, probabilities and pre-activations rounded to bf16
