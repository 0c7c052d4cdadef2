"""The forward kernel's hand-over with its producing warps, replayed on the CPU.

bp_mixed_kernel (csrc/bp_mixed.cu): per stage i (buffer s = i & 1) each
producer (two, or one for stages of one pulse) waits empty[s] for stage i - 2
(from i = 2), writes its pulses' records, tables and copies (PB arrivals on
full[s] between them, one each here), waits full[s], rewrites its windows and
arrives once on ready[s]; each of the 8 accumulating warps waits
ready[s], consumes and arrives on empty[s].  Every wait is a parity wait.
Random interleavings: no deadlock, every wait released by its own stage's
phase, no buffer refilled while a warp still reads it.
"""
import random

import pytest

from test_stage_protocol import Barrier, WARPS


def producer(n, skip_empty=False):
    for i in range(n):
        s = i & 1
        if i >= 2 and not skip_empty:
            yield ("wait", ("empty", s), ((i - 2) >> 1) & 1, i - 2)
        yield ("produce", i)
        yield ("arrive", ("full", s))
        yield ("wait", ("full", s), (i >> 1) & 1, i)
        yield ("rewrite", i)
        yield ("arrive", ("ready", s))


def consumer(n):
    for i in range(n):
        s = i & 1
        yield ("wait", ("ready", s), (i >> 1) & 1, i)
        yield ("consume", i)
        yield ("arrive", ("empty", s))


def replay(n, seed, producers=2, **kw):
    rnd = random.Random(seed)
    count = {"full": producers, "ready": producers, "empty": WARPS}
    bars = {(k, b): Barrier(c) for k, c in count.items() for b in range(2)}
    did = {"full": {}, "ready": {}, "empty": {}}
    progs = [producer(n, **kw) for _ in range(producers)] + [consumer(n) for _ in range(WARPS)]
    op = [next(p) for p in progs]
    live = set(range(len(progs)))
    while live:
        can = [w for w in live if op[w][0] != "wait" or bars[op[w][1]].passed(op[w][2])]
        assert can, f"deadlock: n={n} seed={seed}"
        w = rnd.choice(can)
        what = op[w][0]
        if what == "wait":
            kind, stage = op[w][1][0], op[w][3]
            assert did[kind].get(stage, 0) == count[kind], (kind, stage)
        elif what == "arrive":
            bars[op[w][1]].arrive()
        else:
            stage = op[w][1]
            if what in ("produce", "rewrite") and stage >= 2:
                assert did["empty"].get(stage - 2, 0) == WARPS
            if what == "consume":
                assert did["ready"].get(stage, 0) == producers
            key = {"produce": "full", "rewrite": "ready", "consume": "empty"}[what]
            did[key][stage] = did[key].get(stage, 0) + 1
        try:
            op[w] = next(progs[w])
        except StopIteration:
            live.discard(w)
    assert all(did["empty"].get(i, 0) == WARPS for i in range(n))


@pytest.mark.parametrize("producers", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 12])
def test_hand_over(n, producers):
    for seed in range(200):
        replay(n, seed, producers)


def test_replay_catches_a_missing_empty_wait():
    with pytest.raises(AssertionError):
        for seed in range(200):
            replay(6, seed, skip_empty=True)
