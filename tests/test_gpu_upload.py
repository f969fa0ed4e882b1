"""Uploads into tile buffers of freed weights: values and padding do not depend on what a buffer held before."""
import numpy as np
import pytest

from oracle import oracle as O
from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu


# buffers of one size; of sizes that replace each other once the kept bytes are at their limit (nine of 36 MB); more than are
# kept by number
@pytest.mark.parametrize("rows,k,count", [(272, 1024, 3), (8192, 4096, 9), (16, 32, 300)])
def test_weights_in_used_buffers(rows, k, count):
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    qt = Q.QuantizationType.Q8_0
    ctx, orc = CudaContext(0), O.COracle()
    try:
        big = Q.synth_weight(qt, rows, k, 1)
        held = [QuantizedWeight(ctx, qt, big, rows, k) for _ in range(count)]
        for w in held:
            w.close()
        for r, seed in ((rows, 2), (rows - 5, 3), (rows, 4)):  # the second one leaves padded rows
            blocks = Q.synth_weight(qt, r, k, seed)
            w = QuantizedWeight(ctx, qt, blocks, r, k)
            n = min(r, 64)
            want = orc.dequant(O.Q8_0, blocks[-n:], n * k).reshape(n, k)
            assert np.array_equal(w.dequantize_to_array()[-n:].view(np.uint32), want.view(np.uint32))
            w.close()
    finally:
        ctx.close()


@pytest.mark.parametrize("other_thread", [False, True])
def test_freed_while_a_stream_is_recorded(other_thread):
    """A weight that the recording has nothing to do with: the free succeeds, the recording goes on, its replay is right, and
    an upload afterwards (into the kept buffer, if there is one) disturbs neither."""
    import threading

    from warpforge_b200 import _native as N
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    qt, rows, k = Q.QuantizationType.Q4_0, 512, 1024
    ctx, orc = CudaContext(0), O.COracle()
    try:
        blocks = [Q.synth_weight(qt, rows, k, s) for s in (1, 2)]
        a, b = (QuantizedWeight(ctx, qt, v, rows, k) for v in blocks)
        xb = Q.synth_activation_bf16(1, k, 3)
        dx, dy = ctx.allocate(xb.nbytes), ctx.allocate(rows * 4)
        ctx.copy_to_device(dx, xb)
        call = lambda w, s: ctx._ck("wf_qlinear", ctx._lib.wf_qlinear(ctx.handle, w.handle, dx, N.WF_DTYPE_BF16, 1, 1, dy, 1, s))  # noqa: E731
        call(b, 0)
        s = ctx.create_stream()
        ctx.graph_begin(s)
        call(a, s)
        if other_thread:
            rc = []
            t = threading.Thread(target=lambda: rc.append(ctx._lib.wf_weight_free(ctx.handle, b.handle)))
            t.start()
            t.join()
            assert rc == [N.WF_OK]
            b.handle = 0
        else:
            b.close()
        call(a, s)
        g = ctx.graph_end(s)
        c = QuantizedWeight(ctx, qt, blocks[1], rows, k)
        want = orc.qlinear(O.Q4_0, blocks[0], rows, k, Q.bf16_bits_to_float(xb), nthreads=2)
        got = np.zeros((1, rows), np.float32)
        ctx.copy_to_device(dy, got)
        ctx.graph_launch(g, s)
        ctx.synchronize(s)
        ctx.copy_to_host(got, dy)
        assert np.max(np.abs(got - want)) <= 1e-3 * np.max(np.abs(want))
        assert np.array_equal(c.dequantize_to_array().view(np.uint32), orc.dequant(O.Q4_0, blocks[1], rows * k).reshape(rows, k).view(np.uint32))
        ctx.graph_destroy(g)
        for w in (a, c):
            w.close()
    finally:
        ctx.close()


def test_freed_after_use_on_a_stream_of_another_library():
    """Work on a stream that the context did not create cannot be waited for by itself: the buffer is not kept, and the next
    upload does not write under a kernel that still reads it."""
    import torch

    from warpforge_b200 import _native as N
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    qt, rows, k, m = Q.QuantizationType.Q4_0, 16384, 4096, 512
    ctx = CudaContext(0)
    try:
        one, two = (Q.synth_weight(qt, rows, k, s) for s in (1, 2))
        s = torch.cuda.Stream()
        x, y = torch.randn(m, k, device="cuda").bfloat16(), [torch.empty(m, rows, device="cuda") for _ in range(20)]
        torch.cuda.synchronize()
        w = QuantizedWeight(ctx, qt, one, rows, k)
        for t in y:  # some milliseconds
            N.check("wf_qlinear", ctx._lib.wf_qlinear(ctx.handle, w.handle, x.data_ptr(), N.WF_DTYPE_BF16, 1, m, t.data_ptr(), 1, s.cuda_stream), ctx.handle)
        w.close()
        v = QuantizedWeight(ctx, qt, two, rows, k)
        torch.cuda.synchronize()
        ctx.synchronize(s.cuda_stream)
        assert all(torch.equal(t, y[0]) for t in y)
        v.close()
    finally:
        ctx.close()


def test_kept_buffers_count_as_free_memory():
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    ctx = CudaContext(0)
    try:
        def once():
            QuantizedWeight(ctx, Q.QuantizationType.Q4_0, np.zeros(8192 * 4096 // 32 * 18, np.uint8), 8192, 4096).close()

        once()  # the upload's own buffers
        before = ctx.device_info()["free_mem"]
        w = QuantizedWeight(ctx, Q.QuantizationType.Q4_0, np.zeros(8192 * 4096 // 32 * 18, np.uint8), 8192, 4096)
        assert ctx.device_info()["free_mem"] <= before - w.device_bytes() // 2
        w.close()
        assert ctx.device_info()["free_mem"] >= before
    finally:
        ctx.close()
