"""A recorded graph holds the addresses of the scratch its kernels exchange partial results and converted activations
through.  It must go on giving the same bits after the stream it was recorded on is gone, and after a larger call on that
stream has replaced a buffer; the freed sizes are allocated again and filled meanwhile, so that a graph that still used
them would show it."""
import ctypes

import numpy as np
import pytest

from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu

PAIRS = (784, 11168, 1319, False)
CASES = [  # (rows, k, tokens): clusters, several token tiles, pairs of CTAs, fp32 tokens, sums that go through memory, one token cut between CTAs
    (1000, 1120, 64, False), (3072, 1024, 512, False), PAIRS, (640, 1024, 96, True), (700, 27008, 31, False), (4096, 11008, 1, False)]


def _setup(ctx, rows, k, m, f32):
    from warpforge_b200 import _native as N
    from warpforge_b200.backend import QuantizedWeight

    w = QuantizedWeight(ctx, Q.QuantizationType.Q4_0, Q.synth_q4_0(rows, k, 5), rows, k)
    x = Q.synth_activation_f32(m, k, 6) if f32 else Q.synth_activation_bf16(m, k, 6)
    dx, dy = ctx.allocate(x.nbytes), ctx.allocate(m * rows * 4)
    ctx.copy_to_device(dx, x)
    dtype = N.WF_DTYPE_F32 if f32 else N.WF_DTYPE_BF16
    call = lambda s, m_=m: ctx._ck("wf_qlinear", ctx._lib.wf_qlinear(ctx.handle, w.handle, dx, dtype, 1, m_, dy, 1, s))  # noqa: E731
    return w, dx, dy, call


def _read(ctx, dy, m, rows):
    out = np.empty((m, rows), np.float32)
    ctx.copy_to_host(out, dy)
    return out


def _churn(ctx):
    """Device memory of many sizes, filled."""
    for mb in (1, 2, 8, 16, 40):
        for _ in range(3):
            ctx.copy_to_device(ctx.allocate(mb << 20), np.full(mb << 20, 0xA5, np.uint8))


@pytest.mark.parametrize("rows,k,m,f32", CASES)
def test_stream_destroyed(rows, k, m, f32):
    from warpforge_b200.backend import CudaContext

    ctx = CudaContext(0)
    try:
        if (rows, k, m, f32) == PAIRS:  # whose pieces lie in the stream's scratch
            plan = [ctypes.c_int() for _ in range(5)]
            ctx._ck("plan", ctx._lib.wf_plan_many_tokens(ctx.handle, Q.QuantizationType.Q4_0.ggml_type, rows, k, m, 0, *map(ctypes.byref, plan)))
            assert plan[0].value == 1
        w, dx, dy, call = _setup(ctx, rows, k, m, f32)
        s = ctx.create_stream()
        call(s)  # the scratch of the stream
        ctx.synchronize(s)
        want = _read(ctx, dy, m, rows)
        ctx.graph_begin(s)
        call(s)
        g = ctx.graph_end(s)
        ctx.destroy_stream(s)
        _churn(ctx)
        for _ in range(2):
            ctx.copy_to_device(dy, np.zeros((m, rows), np.float32))
            ctx.graph_launch(g)
            ctx.synchronize()
            assert np.array_equal(_read(ctx, dy, m, rows).view(np.uint32), want.view(np.uint32))
        ctx.graph_destroy(g)
        w.close()
    finally:
        ctx.close()


def test_buffer_replaced_by_a_larger_call():
    from warpforge_b200.backend import CudaContext

    ctx = CudaContext(0)
    try:
        rows, k, m = 1000, 1120, 1500
        w, dx, dy, call = _setup(ctx, rows, k, m, False)
        s, few = ctx.create_stream(), 40
        call(s, few)
        ctx.synchronize(s)
        want = _read(ctx, dy, few, rows)
        ctx.graph_begin(s)
        call(s, few)
        g = ctx.graph_end(s)
        call(s)  # needs more
        ctx.synchronize(s)
        _churn(ctx)
        ctx.copy_to_device(dy, np.zeros((few, rows), np.float32))
        ctx.graph_launch(g, s)
        ctx.synchronize(s)
        assert np.array_equal(_read(ctx, dy, few, rows).view(np.uint32), want.view(np.uint32))
        ctx.graph_destroy(g)
        w.close()
    finally:
        ctx.close()
