"""Host logic of the several-token decode kernel: how a weight is cut into k-slices and warp teams
(`wf_plan_several_tokens`, no device needed).  Every cut must cover K, fit shared memory and the partial-sum
buffer, use a team size the kernel knows, and keep every warp's work within a small factor of the even share."""
import ctypes
import itertools

import pytest

from warpforge_b200 import _native as N

QTYPES = {2: (128, 1152), 3: (128, 1280), 8: (128, 2176), 14: (256, 2368), 6: (128, 2176)}  # ggml type id: (tile k, tile bytes); Q5_0 runs as Q8_0
SHAPES = [(11008, 4096), (4096, 11008), (4096, 4096), (32000, 4096), (44032, 4096), (1024, 8192), (128, 8192), (3584, 8192),
          (1024, 28672), (16, 32), (7, 256), (100000, 256), (64, 131072)]


def _plan(qt, rows, k, cols, f32=0, sms=148):
    s, kc, team, part, smem = ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_int(), ctypes.c_int64()
    rc = N.load().wf_plan_several_tokens(qt, rows, k, cols, f32, sms, ctypes.byref(s), ctypes.byref(kc), ctypes.byref(team),
                                         ctypes.byref(part), ctypes.byref(smem))
    assert rc == N.WF_OK
    return s.value, kc.value, team.value, part.value, smem.value


@pytest.mark.parametrize("qt", sorted(QTYPES))
def test_every_cut_is_valid(qt):
    tk, tb = QTYPES[qt]
    for (rows, k), cols in itertools.product(SHAPES, (1, 3, 4, 8, 9, 16, 17, 30, 32)):
        if k % (256 if qt == 14 else 32):
            continue
        slices, kc, team, part, smem = _plan(qt, rows, k, cols)
        rt, kt = -(-rows // 16), -(-k // tk)
        if slices == 0:  # nothing fits: only allowed when even one slice per k-tile overflows the partial sums
            assert kt * cols * rt * 64 > (8 << 20) or cols * (tk * 2 + 64) > 200 * 1024, (qt, rows, k, cols)
            continue
        assert 1 <= slices <= min(kt, 64, 148) and kc >= 1
        assert (slices - 1) * kc < kt <= slices * kc, "the slices cover K exactly, the last one may be shorter"
        assert team in (1, 2, 3, 4, 5, 8, 16)
        assert smem <= 200 * 1024
        assert part == int(slices > 1)
        if part:
            assert slices * cols * rt * 64 <= (8 << 20)
        # the busiest warp: units of its team x its share of a unit's tiles, against the even share over 148 x 16 warps
        teams = 16 // team
        worst = 0
        for sl in range(slices):
            ctas = (148 - sl + slices - 1) // slices
            kcs = min(kc, kt - sl * kc)
            worst = max(worst, -(-(-(-rt // ctas)) // teams) * -(-kcs // team))
        even = rt * kt / (148 * 16)
        if kt <= 256:  # beyond 64 slices of K (K > 8192 k-tiles' worth per row-tile) the slice count is capped
            assert worst <= max(4.0 * even, even + 3), (qt, rows, k, cols, slices, kc, team, worst, even)


def test_fp32_tokens_always_use_partial_sums_and_bad_arguments_are_refused():
    slices, kc, team, part, _ = _plan(8, 4096, 4096, 3, f32=1)
    assert slices >= 1 and part == 1
    lib = N.load()
    z = ctypes.c_int()
    assert lib.wf_plan_several_tokens(2, 4096, 4096, 33, 0, 148, ctypes.byref(z), ctypes.byref(z), ctypes.byref(z), None, None) == N.WF_ERR_INVALID_ARGUMENT
    assert lib.wf_plan_several_tokens(12, 4096, 4096, 8, 0, 148, ctypes.byref(z), ctypes.byref(z), ctypes.byref(z), None, None) == N.WF_ERR_UNSUPPORTED_TYPE
    assert lib.wf_plan_several_tokens(2, 4096, 4096, 8, 0, 148, None, ctypes.byref(z), ctypes.byref(z), None, None) == N.WF_ERR_INVALID_ARGUMENT


def test_fewer_sms_still_cut_sensibly():
    for sms in (1, 8, 132):
        slices, kc, team, _, smem = _plan(2, 11008, 4096, 8, sms=sms)
        assert 1 <= slices <= sms and smem <= 200 * 1024


def _program_plan(qt, shapes, tokens, sms=148):
    n = len(shapes)
    rows, ks = ((ctypes.c_int64 * n)(*v) for v in zip(*shapes))
    s, kc = (ctypes.c_int * n)(), (ctypes.c_int * n)()
    assert N.load().wf_plan_program(qt, n, rows, ks, tokens, sms, s, kc) == N.WF_OK
    return list(s), list(kc)


@pytest.mark.parametrize("qt", sorted(QTYPES))
def test_a_program_of_like_launches_is_cut_as_a_call_is(qt):
    """Wherever a call runs in clusters or in one slice, a program's launches do, and never with sums through memory, which they do not
    know.  Nothing changes from launch to launch, so with fewer row-tiles than SMs it is the call's own cut; beyond, clusters are
    charged and may give way to one slice."""
    tk, _ = QTYPES[qt]
    rows = [16, 256, 512, 1024, 2560, 4096, 12288, 22016, 44032]
    ks = [512, 1024, 4096, 8448, 9216, 11008, 12288, 16384, 16896, 21248, 22016, 25600, 26880]
    for r, k, tokens in itertools.product(rows, ks, (2, 3, 4, 5, 8)):
        slices, kc = _program_plan(qt, [(r, k)] * 3, tokens)
        call = _plan(qt, r, k, tokens)
        if 1 <= call[0] <= 8:
            assert slices == [call[0]] * 3 or (r >= 148 * 16 and slices == [1] * 3), (qt, r, k, tokens)
        kt = -(-k // tk)
        for s, c in zip(slices, kc):
            assert s == 0 or (s <= 8 and (s - 1) * c < kt <= s * c)


@pytest.mark.parametrize("qt,rows,k,tokens", [(8, 1024, 9216, 4), (14, 1024, 9216, 4), (8, 1024, 9216, 5), (2, 256, 16896, 2), (2, 512, 25600, 2), (8, 1024, 22016, 2)])
@pytest.mark.parametrize("others", [[], [(4096, 4096), (22016, 4096)]])
def test_a_change_that_costs_is_no_reason_to_give_the_launches_up(qt, rows, k, tokens, others):
    slices, _ = _program_plan(qt, [(rows, k)] + others, tokens)
    assert all(1 <= s <= 8 for s in slices)


def test_a_program_that_no_launch_fits_and_bad_arguments():
    assert _program_plan(2, [(4096, 4096), (64, 1 << 20)], 8)[0] == [0, 0]
    one, k = (ctypes.c_int64 * 1)(4096), (ctypes.c_int64 * 1)(4096)
    s, kc = (ctypes.c_int * 1)(), (ctypes.c_int * 1)()
    lib = N.load()
    assert lib.wf_plan_program(2, 1, one, k, 9, 148, s, kc) == N.WF_ERR_INVALID_ARGUMENT
    assert lib.wf_plan_program(2, 0, one, k, 4, 148, s, kc) == N.WF_ERR_INVALID_ARGUMENT
    assert lib.wf_plan_program(12, 1, one, k, 4, 148, s, kc) == N.WF_ERR_UNSUPPORTED_TYPE
