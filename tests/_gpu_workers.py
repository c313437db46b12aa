"""Rank bodies for the multi-GPU tests: one process per GPU over NCCL. Every device-side wait in
the library is bounded, so a protocol error ends as a status (checked with group.check()) or a
mismatch, never as a hang. No test here faults, traps or hangs a GPU on purpose."""

import time

import torch
import torch.distributed as dist

from fast_ulysses_b200 import UlyssesGroup


def ref_even(x, mode, world):
    b, s, n, d = x.shape
    if mode == 0:
        t = x.reshape(b, s, world, n // world, d).permute(2, 0, 1, 3, 4).contiguous()
        o = torch.empty_like(t)
        dist.all_to_all_single(o, t)
        return o.permute(1, 0, 2, 3, 4).reshape(b, world * s, n // world, d)
    t = x.reshape(b, world, s // world, n, d).permute(1, 0, 2, 3, 4).contiguous()
    o = torch.empty_like(t)
    dist.all_to_all_single(o, t)
    return o.permute(1, 2, 0, 3, 4).reshape(b, s // world, world * n, d)


def ref_uneven(x, mode, seq, heads, rank, world):
    b, d = x.shape[0], x.shape[3]
    if mode == 0:
        h0 = [sum(heads[:p]) for p in range(world)]
        send = [x[:, :, h0[p]:h0[p] + heads[p]].contiguous() for p in range(world)]
        recv = [torch.empty(b, seq[p], heads[rank], d, dtype=x.dtype, device=x.device) for p in range(world)]
        dist.all_to_all(recv, send)
        return torch.cat(recv, dim=1)
    s0 = [sum(seq[:p]) for p in range(world)]
    send = [x[:, s0[p]:s0[p] + seq[p]].contiguous() for p in range(world)]
    recv = [torch.empty(b, seq[rank], heads[p], d, dtype=x.dtype, device=x.device) for p in range(world)]
    dist.all_to_all(recv, send)
    return torch.cat(recv, dim=2)


def bits(t):
    return t.contiguous().view(torch.uint8)


def correctness(rank, world):
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    fails = []

    def expect(cond, what):
        if not cond:
            fails.append(what)

    for flags, tag in ((0, "bulk"), (8, "ldst")):
        g._handle.set_test_flags(flags)
        for dtype in (torch.float16, torch.bfloat16):
            for d in (64, 128, 384):
                for mode in (0, 1):
                    torch.manual_seed(100 + rank)
                    shape = (2, 96, 2 * world, d) if mode == 0 else (2, 96 * world, 2, d)
                    x = torch.randn(shape, device=dev, dtype=dtype)
                    y = g.all_to_all_4d(x, mode=mode)
                    expect(torch.equal(y, ref_even(x, mode, world)), f"{tag} even {dtype} d={d} mode={mode}")
        # uneven: near-even and skewed
        for seq, heads in (([97 + p for p in range(world)], [2 + (p % 2) for p in range(world)]),
                           ([5 + 40 * p for p in range(world)], [1 + p for p in range(world)])):
            torch.manual_seed(rank)
            x0 = torch.randn(1, seq[rank], sum(heads), 128, device=dev, dtype=torch.bfloat16)
            y0 = g.all_to_all_4d(x0, mode=0, seq_splits=seq, head_splits=heads)
            expect(torch.equal(y0, ref_uneven(x0, 0, seq, heads, rank, world)), f"{tag} uneven mode 0 {seq}")
            x1 = torch.randn(1, sum(seq), heads[rank], 128, device=dev, dtype=torch.bfloat16)
            y1 = g.all_to_all_4d(x1, mode=1, seq_splits=seq, head_splits=heads)
            expect(torch.equal(y1, ref_uneven(x1, 1, seq, heads, rank, world)), f"{tag} uneven mode 1 {seq}")
            back = g.all_to_all_4d(y0, mode=1, seq_splits=seq, head_splits=heads)
            expect(torch.equal(back, x0), f"{tag} round trip {seq}")
    g._handle.set_test_flags(0)

    # byte dtypes round trip
    for dtype, d in ((torch.float32, 32), (torch.float8_e4m3fn, 64), (torch.float8_e5m2, 64), (torch.int8, 64),
                     (torch.uint8, 64)):
        x = torch.randint(0, 120, (1, 64, 2 * world, d), device=dev).to(dtype)
        y = g.all_to_all_4d(x)
        expect(torch.equal(bits(y), bits(ref_even(bits(x).reshape(1, 64, 2 * world, -1), 0, world))), f"bytes {dtype}")
        expect(torch.equal(bits(g.all_to_all_4d(y, mode=1)), bits(x)), f"round trip {dtype}")

    # out= plain, out=empty_output (zero-copy: internal window untouched), result survives next call
    x = torch.randn(2, 128, 4 * world, 128, device=dev, dtype=torch.bfloat16)
    want = ref_even(x, 0, world)
    plain = torch.empty_like(want)
    expect(g.all_to_all_4d(x, out=plain) is plain and torch.equal(plain, want), "out= plain")
    e_sync = g._handle.epoch_debug(x, 0)
    zc = g.empty_output(x)
    g.all_to_all_4d(x, out=zc)
    expect(torch.equal(zc, want), "out=empty_output")
    expect(g._handle.epoch_debug(zc, 2) == 2 and g._handle.epoch_debug(x, 0) == e_sync, "zero-copy path taken")
    kept = g.all_to_all_4d(x)
    g.all_to_all_4d(torch.zeros_like(x))
    expect(torch.equal(kept, want), "result survives the next call")

    # 20 rounds on one window: +2 phases per call
    e0 = g._handle.epoch_debug(x, 0)
    for _ in range(20):
        g.all_to_all_4d(x)
    expect(g._handle.epoch_debug(x, 0) == e0 + 40, "epoch +2 per call")

    # async: plain, non-contiguous input, out=, lend rotation, off the default stream
    h = g.all_to_all_4d_async(x)
    expect(torch.equal(h.wait(), want), "async")
    xt = torch.randn(2, 4 * world, 128, 128, device=dev, dtype=torch.bfloat16).transpose(1, 2)
    expect(torch.equal(g.all_to_all_4d_async(xt).wait(), ref_even(xt.contiguous(), 0, world)), "async strided")
    o2 = torch.empty_like(want)
    g.all_to_all_4d_async(x, out=o2).wait()
    expect(torch.equal(o2, want), "async out=")
    lent = [g.all_to_all_4d_async(x, lend=True) for _ in range(4)]
    lent = [t.wait() for t in lent]
    expect(len({t.data_ptr() for t in lent}) == 4 and all(torch.equal(t, want) for t in lent), "lend rotation")
    del lent
    side = torch.cuda.Stream(device=dev)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        r = g.all_to_all_4d_async(x).wait()
        expect(torch.equal(r, want), "async off the default stream")
    torch.cuda.current_stream().wait_stream(side)
    # five async calls in flight at once
    many = [g.all_to_all_4d_async(x * (i + 1)) for i in range(5)]
    for i, t in enumerate(many):
        expect(torch.equal(t.wait(), ref_even(x * (i + 1), 0, world)), f"async in flight {i}")

    # autograd: backward is the other mode with the same (unswapped) splits; double backward
    seq, heads = [33 + 3 * p for p in range(world)], [1 + (p % 3) for p in range(world)]
    xg = torch.randn(1, seq[rank], sum(heads), 64, device=dev, requires_grad=True)
    yg = g.all_to_all_4d(xg, seq_splits=seq, head_splits=heads)
    w = torch.randn_like(yg)
    (yg * w).sum().backward()
    expect(torch.equal(xg.grad, g.all_to_all_4d(w, mode=1, seq_splits=seq, head_splits=heads)), "backward")
    import torch.autograd.forward_ad as fwAD

    p_, t_ = torch.randn_like(xg), torch.randn_like(xg)
    with fwAD.dual_level():
        o = g.all_to_all_4d(fwAD.make_dual(p_, t_), seq_splits=seq, head_splits=heads)
        _, tan = fwAD.unpack_dual(o)
    expect(torch.equal(tan, g.all_to_all_4d(t_, seq_splits=seq, head_splits=heads)), "forward-mode tangent")

    # the kernel's own phase timing moves the same bytes
    yt, stages = g._timed(x)
    expect(torch.equal(yt, want) and stages["transfer"] > 0 and len(stages) == 4, "timed")

    # device barrier, then status
    g.barrier()
    g.check()
    failed = torch.tensor([len(fails)], device=dev)
    dist.all_reduce(failed)
    g.destroy()
    assert not fails, fails
    assert failed.item() == 0


def output_pool(rank, world):
    """The copying call hands out pooled symmetric buffers that the peers write directly. Ranks hold
    different numbers of results alive, so they choose different buffers (or none) for the same call."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    h = g._handle
    fails = []

    def expect(cond, what):
        if not cond:
            fails.append(what)

    def call(seed, mode=0):
        torch.manual_seed(seed * 131 + rank)
        shape = (2, 160, 2 * world, 128) if mode == 0 else (2, 160 * world, 2, 128)
        x = torch.randn(shape, device=dev, dtype=torch.bfloat16)
        return g.all_to_all_4d(x, mode=mode), ref_even(x, mode, world)

    expect(h.output_pool(), "pool is on by default")
    held, wants = [], []
    for step in range(6):
        # rank r keeps its first r results alive (at most three): rank 0 always takes the first
        # buffer, the last ranks run out of buffers and fall back to their window
        y, want = call(step, mode=step % 2)
        expect(torch.equal(y, want), f"step {step}")
        if len(held) < min(rank, 3):
            held.append(y)
            wants.append(want)
        for i, (t, w) in enumerate(zip(held, wants)):
            expect(torch.equal(t, w), f"held result {i} after step {step}")
    hits = h.pool_hits()
    # the result of the previous step is still referenced while the next call runs, so a rank that
    # holds two results finds no free buffer every other step, and one that holds three never again
    expect(hits == {0: 6, 1: 6, 2: 4}.get(rank, 3), f"pool hits {hits} on rank {rank}")
    # the zero-copy and the lent paths next to it
    torch.manual_seed(7 + rank)
    x = torch.randn(2, 160, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    out = g.empty_output(x)
    g.all_to_all_4d(x, out=out)
    expect(torch.equal(out, ref_even(x, 0, world)), "out=")
    expect(torch.equal(g.all_to_all_4d_async(x, lend=True).wait(), ref_even(x, 0, world)), "lend")
    # a larger call replaces the pool on every rank together; older results stay valid
    torch.manual_seed(11 + rank)
    xb = torch.randn(2, 400, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    expect(torch.equal(g.all_to_all_4d(xb), ref_even(xb, 0, world)), "grown pool")
    for i, (t, w) in enumerate(zip(held, wants)):
        expect(torch.equal(t, w), f"held result {i} after growth")
    # switched off (on every rank): window + copy-out again
    h.set_output_pool(False)
    y, want = call(99)
    expect(torch.equal(y, want) and h.pool_hits() == hits + 1, "pool off")
    g.barrier()
    g.check()
    failed = torch.tensor([len(fails)], device=dev)
    dist.all_reduce(failed)
    g.destroy()
    assert not fails, fails
    assert failed.item() == 0


def validation_uniform(rank, world):
    """Rejections raise on every rank before the first handshake: the barrier after each case
    would otherwise wait for a rank that went ahead."""
    import pytest

    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    ok = torch.randn(1, 8, 2 * world, 64, device=dev, dtype=torch.bfloat16)

    def rejects(fragment, fn, exc=RuntimeError):
        with pytest.raises(exc, match=fragment):
            fn()
        dist.barrier()

    rejects("must be a CUDA tensor", lambda: g.all_to_all_4d(ok.cpu()))
    rejects("must be 4D", lambda: g.all_to_all_4d(ok[0]))
    rejects("dtype must be", lambda: g.all_to_all_4d(ok.double()))
    rejects("16-byte aligned", lambda: g.all_to_all_4d(ok[..., :4]))
    rejects("mode must be 0 or 1", lambda: g.all_to_all_4d(ok, mode=3))
    rejects("both seq_splits and head_splits", lambda: g.all_to_all_4d(ok, head_splits=[2] * world))
    rejects("but the splits imply", lambda: g.all_to_all_4d(ok, seq_splits=[9] * world, head_splits=[2] * world))
    rejects("must divide world_size",
            lambda: g.all_to_all_4d(torch.randn(1, 8, 2 * world + 1, 64, device=dev, dtype=torch.bfloat16)))
    rejects("moves no data", lambda: g.all_to_all_4d(ok[:, :0]))
    rejects("out has shape", lambda: g.all_to_all_4d(ok, out=torch.empty(1, 8 * world, 3, 64, device=dev,
                                                                         dtype=torch.bfloat16)))
    rejects("out has dtype", lambda: g.all_to_all_4d(ok, out=torch.empty(1, 8 * world, 2, 64, device=dev)))
    rejects("contiguous CUDA tensor", lambda: g.all_to_all_4d(
        ok, out=torch.empty(1, 2, 8 * world, 64, device=dev, dtype=torch.bfloat16).transpose(1, 2)))
    zc = g.empty_output(ok)
    g.all_to_all_4d(ok, out=zc)
    rejects("input overlaps the window", lambda: g.all_to_all_4d(_alias_of(zc, world), out=zc))
    rejects("does not support autograd", lambda: g.all_to_all_4d(ok.clone().requires_grad_(), out=zc))
    rejects("does not support autograd", lambda: g.all_to_all_4d_async(ok.clone().requires_grad_()))
    rejects("not both", lambda: g.all_to_all_4d_async(ok, out=zc, lend=True), ValueError)
    rejects("does not support torch.vmap", lambda: torch.vmap(lambda t: g.all_to_all_4d(t))(ok.unsqueeze(0)))
    # every op of the library refuses a batched input, not only the functional one
    ops = torch.ops.fast_ulysses_b200
    batched = ok.unsqueeze(0)
    rejects("does not support torch.vmap",
            lambda: torch.vmap(lambda t: ops.all_to_all_4d_out(g._handle, t, 0, None, None, zc))(batched))
    rejects("does not support torch.vmap",
            lambda: torch.vmap(lambda t: ops.all_to_all_4d_staged(g._handle, t, 0, None, None, 0, rank, False))(batched))
    rejects("does not support torch.vmap",
            lambda: torch.vmap(lambda t: ops.all_to_all_4d_staged_out(g._handle, t, 0, None, None, zc, 0, rank))(batched))
    rejects("does not support torch.vmap", lambda: torch.vmap(lambda t: ops.empty_output(g._handle, t, 0, None, None))(batched))
    rejects("does not support torch.vmap",
            lambda: torch.vmap(lambda t: ops.all_to_all_4d_timed(g._handle, t, 0, None, None))(batched))
    # batched gradients are vmap over the backward: the same refusal, reached through autograd
    xg = ok.clone().requires_grad_()
    yg = g.all_to_all_4d(xg)
    rejects("does not support torch.vmap",
            lambda: torch.autograd.grad(yg, xg, torch.ones(3, *yg.shape, device=dev, dtype=yg.dtype),
                                        is_grads_batched=True))
    # empty split lists are not "no splits", also once the plan cache is warm for this shape
    g.all_to_all_4d(ok)
    rejects("seq_splits", lambda: g.all_to_all_4d(ok, seq_splits=[], head_splits=[]))
    held = [g.all_to_all_4d_async(ok, lend=True).wait() for _ in range(4)]
    rejects("lent results may be alive at once", lambda: g.all_to_all_4d_async(ok, lend=True))
    del held
    if torch.cuda.device_count() > world:
        other = torch.device("cuda", world)
        rejects("one group serves exactly one device", lambda: g.all_to_all_4d(ok.to(other)))
        rejects("out", lambda: g.all_to_all_4d(ok, out=torch.empty(1, 8 * world, 2, 64, device=other,
                                                                     dtype=torch.bfloat16)))
    g.check()
    g.destroy()
    rejects("has been destroyed", lambda: g.all_to_all_4d(ok))
    rejects("has been destroyed", lambda: g.all_to_all_4d_async(ok))
    rejects("has been destroyed", lambda: g.all_to_all_4d(ok, out=zc))  # the zero-copy path checks too
    rejects("has been destroyed", lambda: g.empty_output(ok))


def _alias_of(zc, world):
    """An input of the right shape (1, 8, 2*world, 64) that lives inside the window behind `zc`."""
    return zc.view(-1)[: 8 * 2 * world * 64].view(1, 8, 2 * world, 64)


def ordering_control(rank, world):
    """Payload visible when the flag arrives. ARMED (closing flag announced before the payload)
    must tear on some rank; CLEAN must not. Uneven shards make rank 0's transfer the longest."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    seq = [60000] + [2000] * (world - 1)
    heads = [4] * world
    x = torch.empty(1, seq[rank], sum(heads), 128, device=dev, dtype=torch.bfloat16)
    out = g.empty_output(x, seq_splits=seq, head_splits=heads)

    def torn_rounds(flags, rounds=24):
        g._handle.set_test_flags(flags)
        torn = 0
        for i in range(rounds):
            v = float(1 + (i % 100))
            x.fill_(v)
            g.all_to_all_4d(x, out=out, seq_splits=seq, head_splits=heads)
            torn += int(not bool(torch.all(out == v)))
        g._handle.set_test_flags(0)
        t = torch.tensor([torn], device=dev)
        dist.all_reduce(t)
        return int(t.item())

    clean = torn_rounds(0)
    armed = torn_rounds(4)  # FU_A2A_EARLY_PUBLISH
    g.check()
    g.destroy()
    assert clean == 0, f"CLEAN phase tore {clean} times"
    if armed == 0:
        print("BLIND: the armed control produced no stale read; the clean result proves less than it should")


def graph_replay(rank, world):
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    x = torch.randn(1, 2048, 4 * world, 128, device=dev, dtype=torch.bfloat16)
    out = g.empty_output(x)
    g.all_to_all_4d(x, out=out)
    torch.cuda.synchronize()
    dist.barrier()
    e0 = g._handle.epoch_debug(out, 2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.all_to_all_4d(x, out=out)
    # control: a replay must move the data by itself. If the capture had recorded nothing, every
    # check below would be comparing `out` with what the eager call above left in it.
    x.fill_(-3.0)
    out.fill_(123.0)
    torch.cuda.synchronize()
    dist.barrier()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.all(out == -3.0), "the captured graph did not run the collective"
    e0 += 2
    ballast = torch.randn(4096, 4096, device=dev)
    for i in range(8):
        x.copy_(torch.full_like(x, float(i + 1)))
        if rank == i % world:
            for _ in range(24):
                ballast @ ballast  # skew one rank
        graph.replay()
        torch.cuda.synchronize()
        assert torch.all(out == float(i + 1)), f"replay {i} tore"
    assert g._handle.epoch_debug(out, 2) == e0 + 16  # exactly two phases per replay
    g.check()
    g.destroy()


def sync_async_coexist(rank, world):
    """Sync and async calls on unordered streams use separate windows. 2000 rounds with a rotating
    slow rank, exact phase counts at the end, and a liveness sample: events on both streams must
    show, in some sampled round, a synchronous call running inside the device life of the
    asynchronous one. If they never overlap the test has not exercised what it is about (BLIND)."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    rounds = 2000
    xs = torch.empty(1, 256, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    big = torch.empty(1, 4096, 2 * world, 128, device=dev, dtype=torch.bfloat16)  # the async payload lasts longer
    cur, comm = torch.cuda.current_stream(dev), g._comm_stream
    bad, overlapped, sampled = 0, 0, 0
    for i in range(rounds):
        a_val, b_val = float(i % 50), float(100 + i % 50)
        b = torch.full_like(xs, b_val)
        sample = i % 100 == 0
        if sample:
            big.fill_(a_val)
            a = big
        else:
            a = torch.full_like(xs, a_val)
        if rank == i % world and i % 10 == 0:
            torch.cuda._sleep(200000)
        if sample:
            a0 = torch.cuda.Event(enable_timing=True)
            a1 = torch.cuda.Event(enable_timing=True)
            s0 = torch.cuda.Event(enable_timing=True)
            s1 = torch.cuda.Event(enable_timing=True)
            a0.record(cur)  # the async call's staging copy and launch are ordered after this point
        h = g.all_to_all_4d_async(a)
        if sample:
            a1.record(comm)
            s0.record(cur)
        y1 = g.all_to_all_4d(b)
        y2 = g.all_to_all_4d(b)
        if sample:
            s1.record(cur)
        ya = h.wait()
        bad += int(not (torch.all(ya == a_val) and torch.all(y1 == b_val) and torch.all(y2 == b_val)))
        if sample:
            torch.cuda.synchronize()
            sampled += 1
            # the sync pair started before the async call ended, and ended after the async call began
            overlapped += int(s0.elapsed_time(a1) > 0 and a0.elapsed_time(s1) > 0)
    torch.cuda.synchronize()
    assert g._handle.epoch_debug(xs, 0) == 4 * rounds and g._handle.epoch_debug(xs, 1) == 2 * rounds
    g.check()
    g.destroy()
    assert bad == 0
    t = torch.tensor([overlapped], device=dev)
    dist.all_reduce(t)
    if int(t.item()) == 0:
        print("BLIND: no sampled round showed the synchronous calls inside the asynchronous call's life")
    elif rank == 0:
        print(f"liveness: {int(t.item())} of {sampled * world} sampled (round, rank) pairs overlapped")


def window_reuse_race(rank, world):
    """A peer's next call must not overwrite a buffer this rank is still reading: the opening
    handshake makes writers wait for readers, where "readers" means everything queued on the
    calling stream. CLEAN: a slow reader on the calling stream is never torn. ARMED: the same slow
    read on a side stream that nothing orders before the next call is outside that guarantee and
    must see the next call's data at least once; if it never does, CLEAN proved nothing (BLIND)."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    x = torch.empty(1, 4096, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    out = g.empty_output(x)
    cur, side = torch.cuda.current_stream(dev), torch.cuda.Stream(device=dev)

    def rounds(armed, n=40):
        torn, snaps = 0, []
        for i in range(n):
            x.fill_(float(i + 1))
            g.all_to_all_4d(x, out=out)
            if armed:
                side.wait_stream(cur)  # the read starts after this call ...
                with torch.cuda.stream(side):
                    torch.cuda._sleep(2_000_000)  # ... late, and nothing makes the next call wait for it
                    snaps.append((out.clone(), float(i + 1)))
            else:
                if rank == i % world:
                    torch.cuda._sleep(2_000_000)  # a slow reader: its read of `out` is queued behind this
                snapshot = out.clone()  # ordered on the caller's stream, before this rank's next call
                torn += int(not bool(torch.all(snapshot == float(i + 1))))
        cur.wait_stream(side)
        torch.cuda.synchronize()
        torn += sum(int(not bool(torch.all(t == v))) for t, v in snaps)
        t = torch.tensor([torn], device=dev)
        dist.all_reduce(t)
        return int(t.item())

    clean = rounds(False)
    armed = rounds(True)
    g.check()
    g.destroy()
    assert clean == 0, f"CLEAN phase tore {clean} times"
    if armed == 0:
        print("BLIND: the unordered side-stream read was never overwritten; the clean result proves less than it should")


def async_input_may_be_overwritten(rank, world):
    """The asynchronous call's default contract: `x` may be overwritten the moment the call returns
    (the call stages a private copy on the caller's stream). Checked with an overwrite queued
    immediately behind the call, a slow rank so that the transfer starts late, many rounds."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    x = torch.empty(1, 2048, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    bad = 0
    for i in range(30):
        v = float(i + 1)
        x.fill_(v)
        if rank == i % world:
            torch.cuda._sleep(1_000_000)
        h = g.all_to_all_4d_async(x)
        x.fill_(-7.0)  # the next writer, on the caller's stream, right behind the call
        bad += int(not bool(torch.all(h.wait() == v)))
    g.check()
    g.destroy()
    assert bad == 0, f"{bad} results saw the overwrite of x"


def copy_engine_transport(rank, world):
    """The asynchronous call on the copy engines against the kernel transport: bit-exact in both
    modes, with even, uneven and empty shards, batches, out= and lent results; ranks that mix the
    two transports; the synchronous call through the same data path; two phases per call."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    torch.manual_seed(100 + rank)
    heads = 2 * world
    uneven_seq = [40 + 8 * p for p in range(world)]
    uneven_seq[-1] = 0  # one empty shard
    uneven_heads = [3] * world
    uneven_heads[0] = 1
    cases = [((1, 96, heads, 128), {}), ((2, 50, heads, 64), {}), ((3, 7, 4 * world, 32), {}),
             ((2, uneven_seq[rank], sum(uneven_heads), 128), {"seq_splits": uneven_seq, "head_splits": uneven_heads})]
    for setting in ("all", "mixed"):
        mine = "copy_engine" if setting == "all" or rank % 2 == 0 else "kernel"
        for shape, kw in cases:
            x = torch.randn(shape, device=dev, dtype=torch.bfloat16)
            g.set_async_transport("kernel")
            want = g.all_to_all_4d_async(x, **kw).wait().clone()
            back_want = g.all_to_all_4d_async(want, mode=1, **kw).wait().clone()
            assert torch.equal(back_want, x), (shape, "round trip of the kernel transport")
            g.set_async_transport(mine)
            got = g.all_to_all_4d_async(x, **kw).wait()
            assert torch.equal(got, want), (setting, shape, "mode 0")
            back = g.all_to_all_4d_async(got, mode=1, **kw).wait()
            assert torch.equal(back, x), (setting, shape, "mode 1")
            out = g.empty_output(x, **kw)
            g.all_to_all_4d_async(x, out=out, **kw).wait()
            assert torch.equal(out, want), (setting, shape, "out= a symmetric buffer")
            plain = torch.empty_like(want)
            g.all_to_all_4d_async(x, out=plain, **kw).wait()
            assert torch.equal(plain, want), (setting, shape, "out= an ordinary tensor")
            lent = g.all_to_all_4d_async(x, lend=True, **kw).wait()
            assert torch.equal(lent, want), (setting, shape, "lent window")
            del lent
    # many rounds with a rotating late rank: the handshakes around the copies must hold
    g.set_async_transport("copy_engine")
    x = torch.empty(1, 1024, heads, 128, device=dev, dtype=torch.bfloat16)
    probe = torch.empty(1, 1024, heads, 128, device=dev, dtype=torch.bfloat16)
    g.all_to_all_4d_async(x.zero_()).wait()
    torch.cuda.synchronize()
    e0 = g._handle.epoch_debug(probe, 1)
    bad = 0
    for i in range(40):
        x.fill_(float(i + 1))
        if rank == i % world:
            torch.cuda._sleep(2_000_000)
        bad += int(not bool(torch.all(g.all_to_all_4d_async(x).wait() == float(i + 1))))
    torch.cuda.synchronize()
    assert bad == 0, f"{bad} rounds delivered something else than that round's payload"
    assert g._handle.epoch_debug(probe, 1) == e0 + 2 * 40, "two phases per call on the asynchronous window"
    # the synchronous call through the same data path (the pool is a device-side choice, so off)
    g.set_output_pool(False)
    g._handle.set_test_flags(128)  # FU_A2A_COPY_ENGINE
    x = torch.randn(2, 64, heads, 128, device=dev, dtype=torch.bfloat16)
    y = g.all_to_all_4d(x)
    g._handle.set_test_flags(0)
    assert torch.equal(y, g.all_to_all_4d(x))
    g.check()
    g.destroy()


def pooled_result_read_on_a_side_stream(rank, world):
    """A pooled result (the default return of all_to_all_4d) read on a side stream: record_stream()
    does nothing for it, the documented rule is to order the side stream before dropping the
    tensor. With that rule followed the read is never torn, whatever the next calls do."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    cur, side = torch.cuda.current_stream(dev), torch.cuda.Stream(device=dev)
    x = torch.empty(1, 2048, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    bad = 0
    for i in range(24):
        v = float(i + 1)
        x.fill_(v)
        y = g.all_to_all_4d(x)
        side.wait_stream(cur)
        with torch.cuda.stream(side):
            torch.cuda._sleep(1_000_000)
            snap = y.clone()
        cur.wait_stream(side)  # the rule: order the reader before the tensor is dropped
        del y
        x.fill_(-1.0)
        for _ in range(3):  # three calls: every pool buffer is handed out again
            g.all_to_all_4d(x)
        bad += int(not bool(torch.all(snap == v)))
    g.check()
    g.destroy()
    assert bad == 0, f"{bad} side-stream reads were torn"


def subgroups_gpu(rank, world):
    """Two sequence-parallel groups side by side (a 2-D mesh). Phase 1: each against
    torch.distributed on its own process group. Phase 2: the two groups go through DIFFERENT
    sequences of shapes, one of them under a growing skew, with empty_output() inside the loop;
    they share nothing, so neither may wait for or disturb the other, and each group's phase
    counter must end at exactly two per call."""
    tp = 2
    sp = world // tp
    groups = [dist.new_group(list(range(t, world, tp))) for t in range(tp)]
    which = rank % tp
    mine = groups[which]
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(mine, device=dev)
    assert g.world_size == sp and g.rank == rank // tp

    def ref(x):
        b, s, n, d = x.shape
        t = x.reshape(b, s, sp, n // sp, d).permute(2, 0, 1, 3, 4).contiguous()
        o = torch.empty_like(t)
        dist.all_to_all_single(o, t, group=mine)
        return o.permute(1, 0, 2, 3, 4).reshape(b, sp * s, n // sp, d)

    for it in range(10):
        x = torch.randn(1, 64 + it, 2 * sp, 128, device=dev, dtype=torch.bfloat16)
        assert torch.equal(g.all_to_all_4d(x), ref(x))
    # phase 2
    g._handle.set_output_pool(False)  # every call through the window: one phase counter to read
    shapes = [(1, 48, 2 * sp, 64), (2, 200, 4 * sp, 128), (1, 1000, 2 * sp, 128), (1, 16, 8 * sp, 32)]
    order = shapes if which == 0 else shapes[::-1]  # opposite orders in the two groups
    # the largest shape first: a window that grows is a new window, whose counter starts again at zero
    g.all_to_all_4d(torch.zeros(max(shapes, key=lambda sh: sh[0] * sh[1] * sh[2] * sh[3]), device=dev,
                                dtype=torch.bfloat16))
    probe = torch.empty(order[0], device=dev, dtype=torch.bfloat16)
    e0 = g._handle.epoch_debug(probe, 0)
    calls = 0
    for it in range(12):
        shape = order[it % len(order)]
        x = torch.randn(shape, device=dev, dtype=torch.bfloat16)
        if which == 1:
            torch.cuda._sleep(100_000 * (it + 1))  # one group falls further and further behind
        want = ref(x)
        assert torch.equal(g.all_to_all_4d(x), want), (which, it, "copying call")
        calls += 1
        if it % 3 == 0:
            out = g.empty_output(x)  # collective inside the loop, on this group only
            g.all_to_all_4d(x, out=out)
            assert torch.equal(out, want), (which, it, "zero-copy call")
    torch.cuda.synchronize()
    assert g._handle.epoch_debug(probe, 0) == e0 + 2 * calls, "phase counter of the synchronous window"
    g.check()
    g.destroy()


def peer_timeout_is_reported(rank, world):
    """Host-made failure: one rank never announces (test flag), the others' bounded waits run out,
    report through check(), and every context stays usable. Runs with plain peer loads/stores."""
    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev, timeout_ms=300)
    x = torch.randn(1, 64, 2 * world, 64, device=dev, dtype=torch.bfloat16)
    g.all_to_all_4d(x)  # window exists, clean round
    g.check()
    dist.barrier()
    if rank == world - 1:
        g._handle.set_test_flags(16)  # FU_A2A_MUTE
    g.all_to_all_4d(x)
    g._handle.set_test_flags(0)
    raised = False
    try:
        g.check()
    except RuntimeError as e:
        raised = "timed out" in str(e) and f"waiting on rank {world - 1}" in str(e)
    # the silent rank itself may or may not have run out of time waiting for the others
    assert raised or rank == world - 1, "the missing announcement was not reported"

    # the fp8 exchange waits no longer than its group does either
    from fast_ulysses_b200.ops import fp8

    x = torch.randn(1, 64, 2 * world, 128, device=dev, dtype=torch.bfloat16)
    fp8.all_to_all_4d_fp8(g, x)
    g.check()
    dist.barrier()
    if rank == world - 1:
        g._handle.set_test_flags(16)  # FU_A2A_MUTE
    t0 = time.monotonic()
    fp8.all_to_all_4d_fp8(g, x)
    torch.cuda.synchronize()
    took = time.monotonic() - t0
    g._handle.set_test_flags(0)
    raised = False
    try:
        g.check()
    except RuntimeError as e:
        raised = "timed out" in str(e) and "fp8 window" in str(e)
    assert raised or rank == world - 1, "the missing announcement was not reported"
    assert took < 5.0, f"waited {took:.1f} s in a group with a limit of 0.3 s"
    assert torch.ones(8, device=dev).sum().item() == 8  # context alive
    dist.barrier()
    g.destroy()


def sp_attention_block(rank, world):
    """The fused sequence-parallel attention block (scatter epilogue, attention, pull prologue)
    against the same block without sequence parallelism on the full sequence; uneven shards."""
    from fast_ulysses_b200.models.attention import UlyssesSelfAttention, reference_attention
    from fast_ulysses_b200.ops import gemm

    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    grid, hidden, heads = (4, 10, 16), 768, (6 if world <= 6 else 8)  # 640 tokens
    total = grid[0] * grid[1] * grid[2]
    seq = [total // world + (1 if p < total % world else 0) for p in range(world)]
    if world > 1:
        seq[0] += 8   # uneven on purpose (and not a multiple of 8: the wgrad contraction length is odd-sized)
        seq[-1] -= 8
    hs = [heads // world + (1 if p < heads % world else 0) for p in range(world)]
    torch.manual_seed(42)  # identical weights on every rank
    attn = UlyssesSelfAttention(g, hidden, heads, grid=grid, seq_splits=seq, head_splits=hs)
    with torch.no_grad():
        attn.gamma_q.add_(0.1 * torch.randn_like(attn.gamma_q))
        attn.gamma_k.add_(0.1 * torch.randn_like(attn.gamma_k))
    x_full = torch.randn(1, total, hidden, device=dev).bfloat16()
    dy_full = torch.randn(1, total, hidden, device=dev).bfloat16()
    s0 = sum(seq[:rank])
    x = x_full[:, s0:s0 + seq[rank]].clone().requires_grad_()
    for _ in range(2):  # twice: the windows are reused, the handshakes must keep them apart
        if x.grad is not None:
            x.grad = None
            attn.zero_grad()
        y = attn(x)
        y.backward(dy_full[:, s0:s0 + seq[rank]])
    gemm.check_errors()
    g.check()

    params = [attn.w_qkv, attn.gamma_q, attn.gamma_k, attn.w_o, attn.b_o]
    xr = x_full.float().requires_grad_()
    pr = [p.detach().float().requires_grad_() for p in params]
    yr = reference_attention(xr, *pr, heads, grid)
    yr.backward(dy_full.float())

    def rel(a, b):
        return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()

    assert rel(y, yr[:, s0:s0 + seq[rank]]) < 2e-2, ("y", rel(y, yr[:, s0:s0 + seq[rank]]))
    assert rel(x.grad, xr.grad[:, s0:s0 + seq[rank]]) < 3e-2, ("dx", rel(x.grad, xr.grad[:, s0:s0 + seq[rank]]))
    for name, p, r in zip(("w_qkv", "gamma_q", "gamma_k", "w_o", "b_o"), params, pr):
        gsum = p.grad.float().clone()
        dist.all_reduce(gsum)
        assert rel(gsum, r.grad) < 4e-2, (name, rel(gsum, r.grad))
    g.destroy()


def fused_block_beside_an_async_exchange(rank, world):
    """The fused attention block (persistent kernels whose CTAs wait on peers) while an asynchronous
    all_to_all_4d of the same group is in flight on the comm stream: both are kernels that wait
    for the same kernel on other ranks, so both must always fit on the device together. Short
    time limit: a wait that could not be satisfied would show in check() within half a second."""
    from fast_ulysses_b200.models.attention import UlyssesSelfAttention
    from fast_ulysses_b200.ops import gemm

    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev, timeout_ms=500)
    grid, hidden, heads = (8, 16, 16 * world), 1024, 8 * world  # 2048 tokens per rank
    torch.manual_seed(3)
    attn = UlyssesSelfAttention(g, hidden, heads, grid=grid, timeout_ms=500)
    x = torch.randn(1, attn.s_local, hidden, device=dev).bfloat16().requires_grad_()
    payload = torch.randn(1, 8192, 4 * world, 128, device=dev, dtype=torch.bfloat16)  # long enough to overlap
    want = ref_even(payload, 0, world)
    bad = 0
    for i in range(12):
        if rank == i % world:
            torch.cuda._sleep(300_000)
        h = g.all_to_all_4d_async(payload)
        y = attn(x)
        y.float().sum().backward()
        bad += int(not torch.equal(h.wait(), want))
    torch.cuda.synchronize()
    gemm.check_errors()
    g.check()
    g.destroy()
    assert bad == 0


def fp8_exchange_fused(rank, world):
    """The one-kernel block-scaled fp8 exchange against its unfused composition (quantise kernel,
    byte exchange, dequantise kernel): identical bits, both modes, even shards and the uneven
    shards of a 40-head model (head splits as even as the world allows, sequence shards drawn
    within 10 % of even from a seed every rank shares)."""
    import random

    from fast_ulysses_b200.ops import fp8

    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    rng = random.Random(2024)
    heads = [40 // world + (1 if p < 40 % world else 0) for p in range(world)]
    base = 600
    seq = [base + rng.randint(-base // 10, base // 10) for _ in range(world)]
    torch.manual_seed(9 + rank)
    cases = [((1, 256, 2 * world, 128), 0, None, None), ((2, 64 * world, 3, 128), 1, None, None),
             ((1, seq[rank], 40, 128), 0, seq, heads), ((1, sum(seq), heads[rank], 128), 1, seq, heads)]
    for shape, mode, ss, hs in cases * 2:  # twice: the window is reused, the handshakes keep the calls apart
        x = (torch.randn(shape, device=dev) * 4).bfloat16()
        fused = fp8.all_to_all_4d_fp8(g, x, mode=mode, seq_splits=ss, head_splits=hs)
        plain = fp8.all_to_all_4d_fp8(g, x, mode=mode, seq_splits=ss, head_splits=hs, fused=False)
        assert torch.equal(fused, plain), (shape, mode)
        exact = g.all_to_all_4d(x, mode=mode, seq_splits=ss, head_splits=hs)
        amax = exact.float().abs().amax(-1, keepdim=True).clamp_min(1e-30)
        assert ((fused.float() - exact.float()).abs() / amax).max() < 0.07  # e4m3: three mantissa bits
    g.check()
    g.destroy()


def dit_stack(rank, world):
    from fast_ulysses_b200.models.dit import DiTStack, reference_forward
    from fast_ulysses_b200.ops import gemm

    dev = torch.device("cuda", rank)
    g = UlyssesGroup(device=dev)
    grid = (2, 8, 16 * world)
    total = grid[0] * grid[1] * grid[2]
    torch.manual_seed(7)
    stack = DiTStack(g, depth=2, hidden=256 * max(1, world // 2), heads=2 * max(1, world // 2), ffn=512, grid=grid)
    hidden = stack.blocks[0].hidden
    x_full = torch.randn(1, total, hidden, device=dev).bfloat16()
    s_local = total // world
    x = x_full[:, rank * s_local:(rank + 1) * s_local].clone().requires_grad_()
    y = stack(x)
    y.float().pow(2).sum().backward()
    stack.allreduce_grads()
    gemm.check_errors()
    g.check()
    xr = x_full.float().requires_grad_()
    yr = reference_forward(stack, xr)
    yr.pow(2).sum().backward()

    def rel(a, b):
        return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()

    sl = slice(rank * s_local, (rank + 1) * s_local)
    assert rel(y, yr[:, sl]) < 3e-2, rel(y, yr[:, sl])
    assert rel(x.grad, xr.grad[:, sl]) < 8e-2, rel(x.grad, xr.grad[:, sl])
    g.destroy()


def nvlink_probe_matches_nvml_oracle(rank, world):
    """nvlink_matrix against an independent pynvml walk over the links, pair by pair; the matrix is
    identical on every rank; the constructor accepts a fully joined group with require_nvlink=True."""
    import fast_ulysses_b200 as fu

    dev = torch.device("cuda", rank)
    devices = list(range(world))
    ours = fu.nvlink_matrix(devices)
    assert fu.nvlink_matrix([0, 999]) is None and fu._C.check_nvlink([0, 999]) == ""  # fails open
    try:
        import pynvml

        pynvml.nvmlInit()
    except Exception:
        print("BLIND: no NVML oracle on this machine")
        return
    if ours is None:
        print("BLIND: the probe could not say")
        return

    def text(v):
        return (v.decode() if isinstance(v, bytes) else v).lower()[-12:]

    on_switch, direct, ids = {}, {}, {}
    for i in devices:
        pr = torch.cuda.get_device_properties(i)
        bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
        h = pynvml.nvmlDeviceGetHandleByPciBusId(bus.encode())
        ids[i] = text(pynvml.nvmlDeviceGetPciInfo(h).busId)
        on_switch[i], direct[i] = False, set()
        for link in range(32):
            try:
                if not pynvml.nvmlDeviceGetNvLinkState(h, link):
                    continue
                kind = pynvml.nvmlDeviceGetNvLinkRemoteDeviceType(h, link)
                if kind == 2:
                    on_switch[i] = True
                elif kind == 0:
                    direct[i].add(text(pynvml.nvmlDeviceGetNvLinkRemotePciInfo(h, link).busId))
            except pynvml.NVMLError:
                continue
    for i in devices:
        for j in devices:
            if i != j:
                want = (on_switch[i] and on_switch[j]) or ids[j] in direct[i]
                assert ours[(i, j)] == want, (i, j, ours[(i, j)], want)
    flat = torch.tensor([int(ours[(i, j)]) for i in devices for j in devices if i != j], device=dev)
    gathered = [torch.zeros_like(flat) for _ in range(world)]
    dist.all_gather(gathered, flat)
    assert all(torch.equal(gathered[0], t) for t in gathered), "the matrix differs between ranks"
    if all(ours.values()):
        g = fu.UlyssesGroup(device=dev, require_nvlink=True)
        g.destroy()
