"""The epilogue of the cluster GEMM (csrc/wf_gemm_split.cuh) when waits run out: four warps meet on two barriers per tile
and wait for the other roles in between; any of those waits may run out in any of the warps, and the CTA's abort flag may
be raised at any moment.  The warps, replayed here under random schedules, must all leave: no warp may stand at a barrier
that another one has left for good.  Deciding in each warp on its own whether to leave (what the loop condition and the
breaks once did) must be caught by the same replay."""
import random

import pytest

WARPS, TILES = 4, 3


def _warp(cta, together, fails):
    """One epilogue warp: yields ("barrier", vote) and gets the barrier's answer, or yields ("step",) anywhere else.
    fails(): whether the wait at hand runs out in this warp."""
    ok, tile = True, 0
    while tile < TILES:
        if together:
            if tile > 0 and not (yield "barrier", ok and not cta["abort"]):
                return
        else:
            if not ok or cta["abort"]:
                return
            if tile > 0:
                yield "barrier", True
        yield "step", None
        if tile > 0 and fails():  # the exchange buffer is free again
            cta["abort"] = True
            if not together:
                return
            ok = False
        if not (yield "barrier", ok):
            return
        for _ in range(2):  # the accumulator; the other ranks' parts
            yield "step", None
            if fails():
                cta["abort"] = True
                ok = False
                break
        if not ok and not together:
            return
        tile += 1


def _replay(seed, together, rate):
    """True when every warp leaves; a schedule in which the remaining warps all stand at a barrier is a hang."""
    rng = random.Random(seed)
    cta = {"abort": False}
    warps = [_warp(cta, together, lambda: rng.random() < rate) for _ in range(WARPS)]
    at = {w: next(g) for w, g in enumerate(warps)}
    while at:
        if rng.random() < rate:
            cta["abort"] = True  # another role of the CTA gives up
        ready = [w for w in at if at[w][0] == "step"]
        if ready:
            moved, answer = [rng.choice(ready)], None
        elif len(at) == WARPS:  # a barrier of 128 threads opens for all four warps only
            moved, answer = list(at), all(v for _, v in at.values())
        else:
            return False
        for w in moved:
            try:
                at[w] = warps[w].send(answer)
            except StopIteration:
                del at[w]
    return True


@pytest.mark.parametrize("rate", [0.0, 0.02, 0.1, 0.4])
def test_all_warps_leave(rate):
    assert all(_replay(s, True, rate) for s in range(3000))


def test_leaving_one_by_one_hangs():
    assert all(_replay(s, False, 0.0) for s in range(100))
    assert not all(_replay(s, False, 0.1) for s in range(3000))
