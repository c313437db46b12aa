"""The GEMM cores' mbarrier pipelines as models, checked over every interleaving of their roles.

`fu::gemm::run` (csrc/kernels/gemm_sm100.cuh; the core of the pulling kernel) has three roles that never share a program counter:
a TMA producer filling a ring of STAGES operand buffers, one MMA thread consuming them into one of
two tensor-memory accumulators, and epilogue warps draining a finished accumulator while the next
tile's main loop already runs. They meet only in mbarriers, and which PHASE PARITY each side waits
for is the part that is easy to get wrong:

    producer   waits  empty[s]           with parity ((it / STAGES) & 1) ^ 1    then fills stage s
    MMA        waits  tmem_empty[acc]    with parity ((tile >> 1) & 1) ^ 1      once per tile
               waits  full[s]            with parity  (it / STAGES) & 1         then reads stage s
               its commit arrives on empty[s]; after the last K-block, on tmem_full[acc]
    epilogue   waits  tmem_full[acc]     with parity  (tile >> 1) & 1           then reads the accumulator
               every epilogue warp arrives on tmem_empty[acc] (count = number of warps)

An mbarrier is modelled as (current phase parity, arrivals still missing); a wait with parity P
passes when the barrier's current phase parity differs from P (the phase with parity P has
completed), which is also why the very first wait on an `empty` barrier, with parity 1, passes at
once. The search explores every interleaving of the role steps for a ring that the K-loop length
does not divide and an odd number of tiles, and checks in every reachable state that

  * the producer never refills a stage the MMA has not read,
  * the MMA reads stage contents in order, and never writes into an accumulator that an epilogue
    warp has yet to drain,
  * the epilogue reads the accumulator of ITS tile, complete,
  * nobody waits for ever.

Negative controls: the same search with the producer's parity un-flipped, and with the accumulator
barrier counting one warp too few, must each find a violation. `run_small` has the same structure on
128 x 128 tiles; its producer also looks at the next stage's barrier while it loads this one and then need not wait for it.

`fu::gemm::run_wide` (pairs of CTAs, two accumulator blocks or one) orders its work differently and is searched
by itself: see `explore_wide`. With one block its operands have a producer each, and both look at the next stage ahead of time.
"""

import pytest


class Bar:
    """mbarrier: phase parity and the arrivals still missing in the current phase."""

    @staticmethod
    def new(count):
        return (0, count, count)

    @staticmethod
    def arrive(b):
        parity, missing, count = b
        return (parity ^ 1, count, count) if missing == 1 else (parity, missing - 1, count)

    @staticmethod
    def passes(b, parity):
        return b[0] != parity


def explore(stages=3, kblocks=2, tiles=3, warps=2, producer_flip=1, empty_count=None, look_flip=None):
    """`look_flip`: the producer looks at the next stage's barrier while it fills this one (None: it does not)."""
    empty_count = warps if empty_count is None else empty_count
    total = tiles * kblocks
    # state: producer it and whether it knows its stage to be free, mma (tile, kb, waiting_acc), epilogue per-warp tile index,
    #        barriers, stage contents, stage consumed marks, accumulator contents and drain marks
    init = ((0, False), (0, 0, True), tuple([0] * warps),
            tuple(Bar.new(1) for _ in range(stages)), tuple(Bar.new(1) for _ in range(stages)),
            (Bar.new(1), Bar.new(1)), (Bar.new(empty_count), Bar.new(empty_count)),
            tuple([-1] * stages), tuple([True] * stages),  # stage holds item, stage has been read
            ((-1, 0), (-1, 0)), ((True,) * warps, (True,) * warps))  # acc = (tile, K-blocks added); drained by warp
    seen, stack = {init}, [init]
    while stack:
        st = stack.pop()
        prod, (m_tile, m_kb, m_wait), e_tiles, full, empty, tfull, tempty, holds, read, acc, drained = st
        p_it, ready = prod
        done = p_it == total and m_tile == tiles and all(t == tiles for t in e_tiles)
        if done:
            continue
        nxt_states = []
        # ---- producer
        if p_it < total:
            s = p_it % stages
            if ready or Bar.passes(empty[s], ((p_it // stages) & 1) ^ producer_flip):
                if not read[s]:
                    return f"producer refills stage {s} (item {holds[s]}) before the MMA has read it"
                h, r, f = list(holds), list(read), list(full)
                h[s], r[s] = p_it, False
                f[s] = Bar.arrive(f[s])
                ahead = p_it + 1
                free = look_flip is not None and Bar.passes(empty[ahead % stages], ((ahead // stages) & 1) ^ look_flip)
                for seen_free in {free, False}:  # it may be looked at before the barrier says so
                    nxt_states.append(((ahead, seen_free), (m_tile, m_kb, m_wait), e_tiles, tuple(f), empty, tfull, tempty,
                                       tuple(h), tuple(r), acc, drained))
        # ---- MMA thread
        if m_tile < tiles:
            a = m_tile & 1
            if m_wait:
                if Bar.passes(tempty[a], ((m_tile >> 1) & 1) ^ 1):
                    if not all(drained[a]):
                        return f"MMA starts tile {m_tile} in accumulator {a} before every epilogue warp has drained tile {acc[a][0]}"
                    ac = list(acc)
                    ac[a] = (m_tile, 0)
                    nxt_states.append((prod, (m_tile, 0, False), e_tiles, full, empty, tfull, tempty, holds, read,
                                       tuple(ac), drained))
            else:
                it = m_tile * kblocks + m_kb
                s = it % stages
                if Bar.passes(full[s], (it // stages) & 1):
                    if holds[s] != it:
                        return f"MMA expects item {it} in stage {s} and finds item {holds[s]}"
                    r, e, ac, tf, dr = list(read), list(empty), list(acc), list(tfull), list(drained)
                    r[s] = True
                    e[s] = Bar.arrive(e[s])  # the commit
                    ac[a] = (m_tile, acc[a][1] + 1)
                    if m_kb + 1 == kblocks:
                        tf[a] = Bar.arrive(tf[a])
                        dr[a] = (False,) * warps
                        nxt_states.append((prod, (m_tile + 1, 0, True), e_tiles, full, tuple(e), tuple(tf), tempty,
                                           holds, tuple(r), tuple(ac), tuple(dr)))
                    else:
                        nxt_states.append((prod, (m_tile, m_kb + 1, False), e_tiles, full, tuple(e), tfull, tempty,
                                           holds, tuple(r), tuple(ac), drained))
        # ---- epilogue warps
        for w in range(warps):
            t = e_tiles[w]
            if t == tiles:
                continue
            a = t & 1
            if Bar.passes(tfull[a], (t >> 1) & 1):
                if acc[a] != (t, kblocks):
                    return f"epilogue warp {w} reads accumulator {a} for tile {t} and finds {acc[a]}"
                et, te, dr = list(e_tiles), list(tempty), list(drained)
                et[w] = t + 1
                te[a] = Bar.arrive(te[a])
                d = list(dr[a])
                d[w] = True
                dr[a] = tuple(d)
                nxt_states.append((prod, (m_tile, m_kb, m_wait), tuple(et), full, empty, tfull, tuple(te), holds, read,
                                   acc, tuple(dr)))
        if not nxt_states:
            return f"deadlock: producer at {p_it}, MMA at {(m_tile, m_kb)}, epilogue at {e_tiles}"
        for n in nxt_states:
            if n not in seen:
                seen.add(n)
                stack.append(n)
    return None


@pytest.mark.parametrize("stages,kblocks,tiles,warps", [(4, 3, 3, 2), (3, 2, 5, 2), (4, 1, 5, 2), (2, 5, 3, 4), (4, 6, 2, 4)])
def test_pipeline_parities_hold_in_every_interleaving(stages, kblocks, tiles, warps):
    assert explore(stages, kblocks, tiles, warps) is None
    assert explore(stages, kblocks, tiles, warps, look_flip=1) is None  # run_small


def test_a_producer_looking_ahead_for_the_wrong_parity_is_found():
    found = explore(3, 2, 3, 2, look_flip=0)
    assert found is not None and "refills" in found


def test_a_producer_waiting_for_the_wrong_parity_is_found():
    found = explore(3, 2, 3, 2, producer_flip=0)
    assert found is not None and ("deadlock" in found or "refills" in found)


def test_an_accumulator_barrier_that_counts_one_warp_too_few_is_found():
    found = explore(3, 2, 5, 2, empty_count=1)
    assert found is not None and ("before every epilogue warp" in found or "finds" in found or "deadlock" in found)


# ---- pairs of CTAs --------------------------------------------------------------------------------------------
def mma_program(items, stages, kblocks, release_early=False):
    """What the issuing warp of `run_wide` does for the blocks (u0, u1) of each item, as in the kernel: the first
    `stages` K-blocks of a tile go into block 0 and then into block 1, and so do the last ones; those
    between, into both. `release_early` gives a stage back after the first block that has read it."""
    ops, stage, phase, uses = [], 0, 0, [0, 0]

    def advance(s, ph):
        return (0, ph ^ 1) if s + 1 == stages else (s + 1, ph)

    for item, (u0, u1) in enumerate(items):
        if u0 == u1:
            continue
        kb = 0
        while kb < kblocks:
            left = kblocks - kb
            if kb > 0 and left > stages and u1 - u0 == 2:
                for _ in range(left - stages):
                    ops += [("wait_full", stage, phase), ("mma", item, 0, kb, stage), ("mma", item, 1, kb, stage), ("empty", stage)]
                    stage, phase = advance(stage, phase)
                    kb += 1
                continue
            run = min(left, stages)
            for u in range(u0, u1):
                if kb == 0:
                    ops.append(("wait_tempty", u, (uses[u] & 1) ^ 1))
                    uses[u] += 1
                s, ph = stage, phase
                for i in range(run):
                    if u == u0:
                        ops.append(("wait_full", s, ph))
                    ops.append(("mma", item, u, kb + i, s))
                    if u + 1 == u1 or release_early:
                        ops.append(("empty", s))
                    s, ph = advance(s, ph)
                if run == left:
                    ops.append(("tfull", u))
            stage, phase = s, ph
            kb += run
    return ops


class Bytes:
    """The mbarrier of a stage: phase parity, whether its bytes have been announced, parts of them that have landed. Parts may land
    before the announcement; the phase completes with both."""

    @staticmethod
    def new():
        return (0, 0, 0)

    @staticmethod
    def add(b, parts, announced, landed):
        parity, a, n = b[0], b[1] + announced, b[2] + landed
        assert a <= 1 and n <= parts, "more than a phase takes"
        return (parity ^ 1, 0, 0) if a == 1 and n == parts else (parity, a, n)


def explore_wide(items, stages=2, kblocks=3, warps=1, flip=1, empty_warps=None, release_early=False, operands=1, look_flip=1, announcers=1):
    """Every interleaving of the producers (one per CTA, or with `operands` = 2 one for each of its operands, which look at the next
    stage while they load this one; a stage is full when the even CTA's first producer has announced all bytes and they have
    landed), the issuing warp of the even CTA, whose commits reach both CTAs, and `warps` epilogue warps per CTA, which all arrive
    on the even CTA's barrier when they have copied a block out. Returns what goes wrong, or None."""
    assert operands == 1 or all(u1 - u0 <= 1 for u0, u1 in items)  # in the kernel, where a pair has one block at a time
    loads = [(n, kb) for n, (u0, u1) in enumerate(items) if u0 != u1 for kb in range(kblocks)]
    blocks = [(n, u) for n, (u0, u1) in enumerate(items) for u in range(u0, u1)]
    ops = mma_program(items, stages, kblocks, release_early)
    total = 2 * warps
    empty_count = total if empty_warps is None else empty_warps
    reads_of = [items[n][1] - items[n][0] for n in range(len(items))]
    parts = 2 * operands  # of a stage, each loaded by a producer of its own
    # producers' positions and what they know of the stage there; MMA program counter, positions of the epilogue warps;
    # full (one barrier, on the even CTA), empty (one per CTA), tmem_full, tmem_empty; what each part of a stage
    # holds and how many blocks have read it; each accumulator's (item, K-blocks added) and who has still to drain it
    init = (((0, False),) * parts, 0, (0,) * total, (Bytes.new(),) * stages, (Bar.new(1),) * stages, (Bar.new(1),) * 2,
            (Bar.new(empty_count),) * 2, ((None, 0),) * (parts * stages), ((-1, 0),) * 2, (0,) * 2)
    seen, stack = {init}, [init]

    def put(t, at, value):
        return t[:at] + (value,) + t[at + 1:]

    while stack:
        prod, pc, epi, full, empty, tfull, tempty, held, acc, todo = stack.pop()
        nxt = []
        for c in range(parts):
            at, ready = prod[c]
            if at < len(loads):
                s, ph = at % stages, ((at // stages) & 1) ^ flip
                if ready or Bar.passes(empty[s], ph):  # the commit reaches both CTAs' barriers at once
                    item, reads = held[parts * s + c]
                    if item is not None and reads < reads_of[item[0]]:
                        return f"producer {c} refills stage {s} ({item}) after {reads} reads"
                    free = operands == 2 and Bar.passes(empty[(at + 1) % stages], (((at + 1) // stages) & 1) ^ look_flip)
                    try:
                        landed = Bytes.add(full[s], parts, int(c < announcers), 1)
                    except AssertionError as e:
                        return f"stage {s}: {e}"
                    for seen_free in {free, False}:  # it may be looked at before the barrier says so
                        nxt.append((put(prod, c, (at + 1, seen_free)), pc, epi, put(full, s, landed), empty, tfull, tempty,
                                    put(held, parts * s + c, (loads[at], 0)), acc, todo))
        if pc < len(ops):
            op = ops[pc]
            state = None
            if op[0] == "wait_full":
                if Bar.passes(full[op[1]], op[2]):
                    state = (prod, pc + 1, epi, full, empty, tfull, tempty, held, acc, todo)
            elif op[0] == "wait_tempty":
                if Bar.passes(tempty[op[1]], op[2]):
                    if todo[op[1]]:
                        return f"the MMA starts block {op[1]} before every epilogue warp has drained it"
                    state = (prod, pc + 1, epi, full, empty, tfull, tempty, held, acc, todo)
            elif op[0] == "mma":
                _, item, u, kb, s = op
                new = held
                for c in range(parts):
                    if held[parts * s + c][0] != (item, kb):
                        return f"the MMA of {(item, u, kb)} finds {held[parts * s + c][0]} in part {c} of stage {s}"
                    new = put(new, parts * s + c, ((item, kb), held[parts * s + c][1] + 1))
                if kb != 0 and acc[u] != (item, kb):
                    return f"the MMA of {(item, u, kb)} adds to {acc[u]}"
                state = (prod, pc + 1, epi, full, empty, tfull, tempty, new, put(acc, u, (item, kb + 1)), todo)
            elif op[0] == "empty":
                state = (prod, pc + 1, epi, full, put(empty, op[1], Bar.arrive(empty[op[1]])), tfull, tempty, held, acc, todo)
            else:
                state = (prod, pc + 1, epi, full, empty, put(tfull, op[1], Bar.arrive(tfull[op[1]])), tempty, held, acc,
                         put(todo, op[1], total))
            if state is not None:
                nxt.append(state)
        for w in range(total):
            if epi[w] < len(blocks):
                item, u = blocks[epi[w]]
                uses = sum(1 for b in blocks[:epi[w]] if b[1] == u)
                if Bar.passes(tfull[u], uses & 1):
                    if acc[u] != (item, kblocks):
                        return f"epilogue warp {w} reads block {u} for item {item} and finds {acc[u]}"
                    nxt.append((prod, pc, put(epi, w, epi[w] + 1), full, empty, tfull, put(tempty, u, Bar.arrive(tempty[u])), held, acc,
                                put(todo, u, todo[u] - 1)))
        if not nxt and (pc < len(ops) or min(prod)[0] < len(loads) or min(epi) < len(blocks)):
            return f"deadlock: producers at {prod}, MMA at {ops[pc:pc + 1]}, epilogue at {epi}"
        for n in nxt:
            if n not in seen:
                seen.add(n)
                stack.append(n)
    return None


WHOLE, FIRST, SECOND, OUTSIDE = (0, 2), (0, 1), (1, 2), (1, 1)


# K shorter than the ring, as long, one more, twice, and with K-blocks in the middle of a tile; whole tiles, then
# single blocks of them, some outside the result
@pytest.mark.parametrize("stages,kblocks", [(2, 1), (2, 2), (2, 3), (2, 4), (2, 6), (3, 2), (3, 5), (3, 7)])
@pytest.mark.parametrize("items", [(WHOLE, WHOLE, WHOLE), (WHOLE, FIRST, SECOND), (FIRST, WHOLE), (WHOLE, SECOND, OUTSIDE, FIRST),
                                   (SECOND, FIRST, SECOND)])
def test_two_blocks_of_a_pair_hold_in_every_interleaving(stages, kblocks, items):
    assert explore_wide(items, stages, kblocks) is None


# one block per pair: its accumulators alternate between the halves of tensor memory
@pytest.mark.parametrize("stages,kblocks", [(2, 1), (2, 3), (3, 2), (3, 4)])
def test_alternating_blocks_of_a_pair_hold_in_every_interleaving(stages, kblocks):
    assert explore_wide((FIRST, SECOND, FIRST, SECOND, FIRST), stages, kblocks) is None


# the same with a producer for each operand: two announce nothing, and all may know from looking ahead that a stage is free
@pytest.mark.parametrize("stages,kblocks,items", [(2, 1, (FIRST, SECOND, FIRST)), (2, 3, (FIRST, SECOND)), (3, 2, (FIRST, SECOND, FIRST)), (3, 4, (FIRST, OUTSIDE, SECOND))])
def test_a_producer_for_each_operand_holds_in_every_interleaving(stages, kblocks, items):
    assert explore_wide(items, stages, kblocks, operands=2) is None


# looking for the wrong parity; both operands of the even CTA announced; none
@pytest.mark.parametrize("fault,text", [(dict(look_flip=0), ("refills",)), (dict(announcers=2), ("more than a phase", "finds")), (dict(announcers=0), ("deadlock",))])
def test_faults_of_the_operands_producers_are_found(fault, text):
    found = explore_wide((FIRST, SECOND, FIRST), 2, 3, operands=2, **fault)
    assert found is not None and any(t in found for t in text), found


@pytest.mark.parametrize("fault,text", [(dict(flip=0), ("deadlock", "refills")), (dict(empty_warps=1), ("before every", "finds", "adds", "deadlock")),
                                        (dict(release_early=True), ("refills", "finds", "deadlock"))])
def test_faults_of_the_pair_schedule_are_found(fault, text):
    found = explore_wide((WHOLE, WHOLE, WHOLE), 2, 3, **fault)
    assert found is not None and any(t in found for t in text), found
