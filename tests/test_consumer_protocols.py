"""The hand-overs of the adjoint and the FP64 kernel, replayed on the CPU.

bp_adjoint_kernel (csrc/bp_adjoint.cu): as the forward kernel's (one or two
producers, see test_producer_protocol.py), but before it refills buffer s = i & 1
a producer waits empty[s] for stage i - 2 and reads that stage's records and the
8 warps' sums (finish); after the last stage it finishes the last two.

bp_fp64_kernel (csrc/bp_fp64.cu): 8 warps, all of which consume; warp 0 also
refills: at stage i it waits empty[s ^ 1] for stage i - 1 (from i = 1), issues
stage i + 1 into buffer s ^ 1 (PB arrivals on full, one here), then waits full[s]
like every warp, consumes and arrives on empty[s].

Random interleavings: no deadlock, every wait released by its own stage's phase,
no buffer, record or sum overwritten while another warp still needs it.
"""
import random

import pytest

from test_stage_protocol import Barrier, WARPS


def adjoint_producer(n, early_refill=False):
    fin = 0
    for i in range(n):
        s = i & 1
        if early_refill and i >= 2:
            yield ("do", "produce", i)
        if i >= 2:
            yield ("wait", ("empty", s), ((i - 2) >> 1) & 1, i - 2)
            yield ("do", "finish", fin)
            fin += 1
        if not (early_refill and i >= 2):
            yield ("do", "produce", i)
        yield ("arrive", ("full", s))
        yield ("wait", ("full", s), (i >> 1) & 1, i)
        yield ("do", "rewrite", i)
        yield ("arrive", ("ready", s))
    for i in range(0 if n < 2 else n - 2, n):
        yield ("wait", ("empty", i & 1), (i >> 1) & 1, i)
        yield ("do", "finish", fin)
        fin += 1


def adjoint_consumer(n):
    for i in range(n):
        s = i & 1
        yield ("wait", ("ready", s), (i >> 1) & 1, i)
        yield ("do", "consume", i)
        yield ("arrive", ("empty", s))


def fp64_warp(n, warp, no_wait=False):
    if warp == 0:
        yield ("do", "produce", 0)
        yield ("arrive", ("full", 0))
    for i in range(n):
        s = i & 1
        if warp == 0 and i + 1 < n:
            if i >= 1 and not no_wait:
                yield ("wait", ("empty", s ^ 1), ((i - 1) >> 1) & 1, i - 1)
            yield ("do", "produce", i + 1)
            yield ("arrive", ("full", s ^ 1))
        yield ("wait", ("full", s), (i >> 1) & 1, i)
        yield ("do", "consume", i)
        yield ("arrive", ("empty", s))


def replay(n, seed, progs, counts, producers, adjoint):
    rnd = random.Random(seed)
    bars = {(k, b): Barrier(c) for k, c in counts.items() for b in range(2)}
    did = {}  # (action, stage) -> warps that have done it
    action_of = {"full": "produce", "ready": "rewrite", "empty": "consume"}
    op = [next(p) for p in progs]
    live = set(range(len(progs)))
    while live:
        can = [w for w in live if op[w][0] != "wait" or bars[op[w][1]].passed(op[w][2])]
        assert can, f"deadlock: n={n} seed={seed}"
        w = rnd.choice(can)
        what = op[w][0]
        if what == "wait":
            kind, stage = op[w][1][0], op[w][3]
            assert did.get((action_of[kind], stage), 0) == counts[kind], (kind, stage)
        elif what == "arrive":
            bars[op[w][1]].arrive()
        else:
            action, stage = op[w][1], op[w][2]
            if action in ("produce", "rewrite") and stage >= 2:
                # the buffer's last stage: consumed by every warp, and this producer's own pulses of it finished
                assert did.get(("consume", stage - 2), 0) == WARPS
                assert not adjoint or did.get(("finish", stage - 2, w), 0) == 1
            if action == "consume":
                need = "rewrite" if adjoint else "produce"
                assert did.get((need, stage), 0) == producers
                # the sums of the buffer's last stage have been read
                assert not adjoint or stage < 2 or did.get(("finish", stage - 2), 0) == producers
            if action == "finish":
                assert did.get(("consume", stage), 0) == WARPS
                did[("finish", stage, w)] = 1
            did[(action, stage)] = did.get((action, stage), 0) + 1
        try:
            op[w] = next(progs[w])
        except StopIteration:
            live.discard(w)
    assert all(did.get(("consume", i), 0) == WARPS for i in range(n))
    assert not adjoint or all(did.get(("finish", i), 0) == producers for i in range(n))


def run_adjoint(n, seed, producers, **kw):
    progs = [adjoint_producer(n, **kw) for _ in range(producers)] + [adjoint_consumer(n) for _ in range(WARPS)]
    replay(n, seed, progs, {"full": producers, "ready": producers, "empty": WARPS}, producers, True)


def run_fp64(n, seed, **kw):
    progs = [fp64_warp(n, w, **kw) for w in range(WARPS)]
    replay(n, seed, progs, {"full": 1, "empty": WARPS}, 1, False)


@pytest.mark.parametrize("producers", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 12])
def test_adjoint_hand_over(n, producers):
    for seed in range(200):
        run_adjoint(n, seed, producers)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 12])
def test_fp64_hand_over(n):
    for seed in range(200):
        run_fp64(n, seed)


def test_replays_catch_an_early_refill():
    with pytest.raises(AssertionError):
        for seed in range(200):
            run_adjoint(6, seed, 2, early_refill=True)
    with pytest.raises(AssertionError):
        for seed in range(200):
            run_fp64(6, seed, no_wait=True)
