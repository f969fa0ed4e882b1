"""Inf and NaN activations through the decode kernels.

One token: the staging writes every activation as digits of a common exponent per 32-k block, and a block with an Inf or a NaN takes a way of
its own.  A lone Inf gives the Inf of the weight's sign (NaN where the weight is zero), as the sum of products does; a NaN gives
NaN; a block with Infs of both signs gives NaN.  Q4_1 and Q4_K multiply codes and offsets apart, so that an Inf may become NaN there.  Rows with finite activations only are the same bits beside such rows (2 - 32 tokens)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from warpforge_b200 import _native as N
from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu

OQ = {"Q4_0": O.Q4_0, "Q4_1": O.Q4_1, "Q5_0": O.Q5_0, "Q8_0": O.Q8_0, "Q4_K": O.Q4_K}
ROWS = 272
INF, NAN = np.float32(np.inf), np.float32(np.nan)


def _k(qname):
    return 1280 if qname == "Q4_K" else 2784  # 2784: the last unit of 128 k holds three blocks


@pytest.fixture(scope="module")
def ctx():
    from warpforge_b200.backend import CudaContext

    c = CudaContext(0)
    yield c
    c.close()


def _upload(ctx, a):
    d = ctx.allocate(a.nbytes)
    ctx.copy_to_device(d, a)
    return d


def _weight(ctx, oracle, qname, rows, k, seed):
    from warpforge_b200.backend import QuantizedWeight

    qt = Q.QuantizationType[qname]
    blocks = Q.synth_weight(qt, rows, k, seed)
    return QuantizedWeight(ctx, qt, blocks, rows, k), oracle.dequant(OQ[qname], blocks, rows * k).reshape(rows, k)


def _same_specials(qname, got, want):
    """NaN where the sum of products has NaN, an Inf of the same sign where it has one, finite elsewhere."""
    if qname in ("Q4_1", "Q4_K"):
        assert np.array_equal(np.isfinite(got), np.isfinite(want)) and np.isnan(got[np.isnan(want)]).all()
        return
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(np.isinf(got), inf)
    assert np.array_equal(np.sign(got[inf]), np.sign(want[inf]))


def _product(w, x):
    with np.errstate(invalid="ignore"):
        return (w.astype(np.float64) * x.astype(np.float64)).sum(-1)


def _qlinear(ctx, w, x, dtype):
    bits = np.ascontiguousarray(x) if dtype == N.WF_DTYPE_F32 else (np.ascontiguousarray(x).view(np.uint32) >> 16).astype(np.uint16)
    m = len(x)
    dx, dy = _upload(ctx, bits), ctx.allocate(m * w.rows * 4)
    ctx._ck("q", ctx._lib.wf_qlinear(ctx.handle, w.handle, dx, dtype, 1, m, dy, 1, 0))
    ctx.synchronize()
    y = np.empty((m, w.rows), np.float32)
    ctx.copy_to_host(y, dy)
    ctx.free(dx)
    ctx.free(dy)
    return y


def _specials(k):
    """(elements set, whether the sum of products says what to expect)"""
    last = k - 32
    yield {k - 1: INF}, True
    yield {0: -INF}, True
    yield {last + 5: INF}, True
    yield {64 + 9: INF, last + 2: INF}, True  # two blocks
    for t in range(4):  # each of the four threads that stage a block, first and last element
        yield {32 * 7 + 8 * t: NAN}, True
        yield {32 * 6 + 8 * t + 7: -NAN}, True
    yield {40: INF, 41: NAN}, True
    yield {96: INF, 127: -INF}, False  # both signs in a block: NaN, whatever the weights' signs


@pytest.mark.parametrize("qname", sorted(OQ))
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_one_token(ctx, oracle, qname, dtype):
    k = _k(qname)
    w, wf = _weight(ctx, oracle, qname, ROWS, k, 11)
    for put, exact in _specials(k):
        x = Q.bf16_bits_to_float(Q.synth_activation_bf16(1, k, 12)).reshape(1, k).astype(np.float32)
        for i, v in put.items():
            x[0, i] = v
        got = _qlinear(ctx, w, x, N.WF_DTYPE_BF16 if dtype == "bf16" else N.WF_DTYPE_F32)[0]
        if exact:
            _same_specials(qname, got, _product(wf, x[0]))
        else:
            assert np.isnan(got).all()
    w.close()


@pytest.mark.parametrize("qname", sorted(OQ))
@pytest.mark.parametrize("m,dtype", [(4, "bf16"), (16, "bf16"), (32, "bf16"), (4, "f32"), (10, "f32")])
def test_several_tokens(ctx, oracle, qname, m, dtype):
    """The affected tokens have no finite output, the others the bits they have without them."""
    k = _k(qname)
    w, _ = _weight(ctx, oracle, qname, ROWS, k, 13)
    clean = Q.bf16_bits_to_float(Q.synth_activation_bf16(m, k, 14)).reshape(m, k).astype(np.float32)
    x = clean.copy()
    x[0, k - 1], x[2, 7], x[m - 1, 33] = INF, NAN, -INF
    d = N.WF_DTYPE_BF16 if dtype == "bf16" else N.WF_DTYPE_F32
    a, b = _qlinear(ctx, w, clean, d), _qlinear(ctx, w, x, d)
    hit = [0, 2, m - 1]
    keep = [i for i in range(m) if i not in hit]
    assert np.isfinite(a).all() and not np.isfinite(b[hit]).any()
    assert np.array_equal(a[keep].view(np.uint32), b[keep].view(np.uint32))
    w.close()


def _program(ctx, w, x, kind, aux, eps):
    """Two projections of one staged row (the group kernel) and their outputs."""
    n, lib = len(w), ctx._lib
    arr = lambda v, t: (t * n)(*v)  # noqa: E731
    ys = [ctx.allocate(ROWS * 4) for _ in w]
    prog = ctypes.c_int64()
    flags = [N.WF_OP_NEW_X | N.WF_OP_DEPENDS] + [0] * (n - 1)
    ctx._ck("create", lib.wf_program_create_fused(
        ctx.handle, n, arr([v.handle for v in w], ctypes.c_int64), arr([x] * n, ctypes.c_int64), arr(ys, ctypes.c_int64), arr(flags, ctypes.c_int),
        arr([kind] * n, ctypes.c_int), arr([aux] * n, ctypes.c_int64), arr([eps] * n, ctypes.c_float), arr([0] * n, ctypes.c_int64), 1, 1, 0, None,
        ctypes.byref(prog)))
    before = ctx.launch_count()
    ctx._ck("run", lib.wf_program_run(ctx.handle, prog.value, 0))
    ctx.synchronize()
    assert ctx.launch_count() - before == 1
    out = [np.empty(ROWS, np.float32) for _ in w]
    for a, p in zip(out, ys):
        ctx.copy_to_host(a, p)
        ctx.free(p)
    ctx._ck("destroy", lib.wf_program_destroy(ctx.handle, prog.value))
    return out


@pytest.mark.parametrize("qname", sorted(OQ))
@pytest.mark.parametrize("kind", ["bf16", "f32", "rmsnorm", "swiglu"])
def test_one_token_program(ctx, oracle, qname, kind):
    k = _k(qname)
    ws, wfs = zip(*(_weight(ctx, oracle, qname, ROWS, k, 15 + i) for i in range(2)))
    base = Q.bf16_bits_to_float(Q.synth_activation_bf16(1, k, 16)).reshape(k).astype(np.float32)
    other = (1 + np.abs(Q.bf16_bits_to_float(Q.synth_activation_bf16(1, k, 17)).reshape(k))).astype(np.float32)
    for put, exact in _specials(k):
        x, aux = base.copy(), other.copy()
        for i, v in put.items():
            (aux if kind in ("rmsnorm", "swiglu") else x)[i] = v  # the operand that does not steer the whole row
        staged = {"bf16": lambda: x, "f32": lambda: x, "rmsnorm": lambda: x / np.sqrt(np.mean(x * x) + 1e-5) * aux,
                  "swiglu": lambda: x / (1 + np.exp(-x)) * aux}[kind]()
        bits = (x.view(np.uint32) >> 16).astype(np.uint16) if kind == "bf16" else x
        code = {"bf16": 0, "f32": N.WF_X_F32, "rmsnorm": N.WF_X_RMSNORM_F32, "swiglu": N.WF_X_SWIGLU_F32}[kind]
        dx, da = _upload(ctx, bits), _upload(ctx, aux)
        got = _program(ctx, ws, dx, code, da if kind in ("rmsnorm", "swiglu") else 0, 1e-5)
        both = any(np.isposinf(v).any() and np.isneginf(v).any() for v in staged.reshape(-1, 32))  # the other factor has signs of its own
        for g, wf in zip(got, wfs):
            if exact:
                _same_specials(qname, g, _product(wf, staged))
            else:
                assert (np.isnan(g) if both else ~np.isfinite(g)).all()
        ctx.free(dx)
        ctx.free(da)
    if kind == "rmsnorm":  # in x itself: the norm is Inf or NaN, every row's answer NaN
        for v in (INF, NAN):
            x = base.copy()
            x[k // 2] = v
            dx, da = _upload(ctx, x), _upload(ctx, other)
            for g in _program(ctx, ws, dx, N.WF_X_RMSNORM_F32, da, 1e-5):
                assert np.isnan(g).all()
            ctx.free(dx)
            ctx.free(da)
    for w in ws:
        w.close()
