"""The ways a several-token product takes from its warps' sums to y: one slice (straight to y, or through shared memory for
fp32 tokens), a cluster of slices in one and in several batches of row-tiles, and partial sums in memory where eight slices
do not fit; the last slice and the last batch shorter than the others, fewer tiles than warps.

Weights are the codes themselves (unit scales) and activations small multiples of a power of two, so every product and every
partial sum is a multiple of 2^-9 below 2^15: exact in fp32 however the additions are ordered.  fp32 tokens need their second
bf16 part."""
import numpy as np
import pytest

from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,m,f32", [
    (16, 32, 2, False), (50, 96, 9, False), (4700, 2048, 8, False),     # one slice
    (260, 2080, 16, False), (7000, 2560, 31, False), (3100, 11008, 17, False),  # clusters; several batches
    (30, 65536, 32, False), (700, 27008, 31, False),                    # memory
    (9000, 1024, 2, True), (3001, 4128, 10, True), (100, 3200, 5, True),
])
def test_exact(rows, k, m, f32):
    from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS, NvidiaBackend, Tensor

    rng = np.random.default_rng(rows + k + m)
    codes = rng.integers(0, 16, (rows, k), dtype=np.uint8)
    blocks = np.zeros((rows, k // 32, 18), np.uint8)
    blocks[:, :, 0:2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
    c = codes.reshape(rows, k // 32, 32)
    blocks[:, :, 2:] = c[:, :, 0::2] | (c[:, :, 1::2] << 4)
    # |y| <= 8 K max|x| stays below 2^15
    x = (rng.integers(-511, 512, (m, k)) / 512.0 if f32 else rng.integers(-8, 9, (m, k)) / 128.0).astype(np.float32)
    backend = NvidiaBackend(0)
    w = backend.upload_weight(Q.QuantizationType.Q4_0, blocks.reshape(rows, -1), rows, k)
    t = Tensor.from_float_array(x) if f32 else Tensor.from_bf16_bits(Q.float_to_bf16_bits(x).reshape(m, k))
    got = [backend.execute(DotGeneralOp(LINEAR_DIMS, (m, rows)), [t, w])[0].data for _ in range(2)]
    want = x.astype(np.float64) @ (codes.astype(np.float64) - 8.0).T
    w.close()
    backend.close()
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want)


@pytest.mark.parametrize("m", [1, 2, 7])
@pytest.mark.parametrize("ks,shared", [
    ((1024,) * 6, (0, 1, 1, 1, 1, 1)),      # six weights on one input: two launches
    ((2080, 2080, 96, 3232), (0, 1, 0, 0)),  # groups of two, one and one
    ((8192, 8192), (0, 1)),                  # several slices at seven tokens
    ((1024, 512), (0, 1)),                   # the second reads the first half of what the first staged: the persistent kernel
])
def test_program_of_one_rank(m, ks, shared):
    """A program's projections, joined where they read the same activations; exact as above."""
    import ctypes

    from warpforge_b200 import _native as N
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    rng = np.random.default_rng(len(ks) + m)
    ctx = CudaContext(0)
    arr = lambda v, t: (t * len(v))(*v)
    ws, xs, ys, want = [], [], [], []
    for i, (k, same) in enumerate(zip(ks, shared)):
        rows = (16, 5000, 33, 700, 1, 2368)[i]
        codes = rng.integers(0, 16, (rows, k), dtype=np.uint8)
        blocks = np.zeros((rows, k // 32, 18), np.uint8)
        blocks[:, :, 0:2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8)
        c = codes.reshape(rows, k // 32, 32)
        blocks[:, :, 2:] = c[:, :, 0::2] | (c[:, :, 1::2] << 4)
        ws.append(QuantizedWeight(ctx, Q.QuantizationType.Q4_0, blocks.reshape(rows, -1), rows, k))
        if not same:
            x = (rng.integers(-8, 9, (m, k)) / 128.0).astype(np.float32)
            bits = Q.float_to_bf16_bits(x).reshape(m, k)
            d = ctx.allocate(bits.nbytes)
            ctx.copy_to_device(d, bits)
        xs.append(d)
        ys.append(ctx.allocate(m * rows * 4))
        want.append(x[:, :k].astype(np.float64) @ (codes.astype(np.float64) - 8.0).T)
    flags = [0 if same else N.WF_OP_NEW_X | (N.WF_OP_DEPENDS if i else 0) for i, same in enumerate(shared)]
    prog = ctypes.c_int64()
    try:
        ctx._ck("create", ctx._lib.wf_program_create(ctx.handle, len(ws), arr([w.handle for w in ws], ctypes.c_int64), arr(xs, ctypes.c_int64),
                                                     arr(ys, ctypes.c_int64), arr(flags, ctypes.c_int), m, 1, 0, None, ctypes.byref(prog)))
        for _ in range(2):
            ctx._ck("run", ctx._lib.wf_program_run(ctx.handle, prog.value, 0))
        ctx.synchronize()
        for y, w in zip(ys, want):
            got = np.empty(w.shape, np.float32)
            ctx.copy_to_host(got, y)
            assert np.array_equal(got, w)
        ctx._ck("destroy", ctx._lib.wf_program_destroy(ctx.handle, prog.value))
    finally:
        ctx.close()


@pytest.mark.parametrize("d,ffn", [(512, 736), (96, 32), (256, 5024)])
def test_swiglu_between_launches(d, ffn):
    """silu(gate) * up made by the launch of a gate and an up projection, in that order, or (up first) by the staging of the
    projection that reads it: the same float operations on gate and up rows whose sums are cut between warps at other places
    (as between the program and the per-projection kernels: 1e-5 of the output scale)."""
    import ctypes

    from warpforge_b200 import _native as N
    from warpforge_b200.backend import CudaContext, QuantizedWeight

    ctx = CudaContext(0)
    arr = lambda v, t: (t * len(v))(*v)
    qt = Q.QuantizationType.Q8_0
    try:
        gate, up = (QuantizedWeight(ctx, qt, Q.synth_weight(qt, ffn, d, s), ffn, d) for s in (1, 2))
        down = QuantizedWeight(ctx, qt, Q.synth_weight(qt, d, ffn, 3), d, ffn)
        x = Q.synth_activation_f32(1, d, 4)
        dx, yg, yu, yd = ctx.allocate(x.nbytes), ctx.allocate(ffn * 4), ctx.allocate(ffn * 4), ctx.allocate(d * 4)
        ctx.copy_to_device(dx, x)
        outs = []
        for first, second in (((gate, yg), (up, yu)), ((up, yu), (gate, yg))):
            prog = ctypes.c_int64()
            ctx._ck("create", ctx._lib.wf_program_create_fused(
                ctx.handle, 3, arr([first[0].handle, second[0].handle, down.handle], ctypes.c_int64), arr([dx, dx, yg], ctypes.c_int64),
                arr([first[1], second[1], yd], ctypes.c_int64), arr([N.WF_OP_NEW_X, 0, N.WF_OP_NEW_X | N.WF_OP_DEPENDS], ctypes.c_int),
                arr([1, 1, 3], ctypes.c_int), arr([0, 0, yu], ctypes.c_int64), None, None, 1, 1, 0, None, ctypes.byref(prog)))
            for _ in range(2):
                ctx._ck("run", ctx._lib.wf_program_run(ctx.handle, prog.value, 0))
            ctx.synchronize()
            outs.append([np.empty(n, np.float32) for n in (ffn, ffn, d)])
            for a, p in zip(outs[-1], (yg, yu, yd)):
                ctx.copy_to_host(a, p)
            ctx._ck("destroy", ctx._lib.wf_program_destroy(ctx.handle, prog.value))
        assert np.isfinite(outs[0][2]).all() and np.any(outs[0][2])
        for a, b in zip(*outs):
            assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b))
    finally:
        ctx.close()


@pytest.mark.parametrize("rows,k,m,f32", [
    (36000, 3072, 32, False),   # clusters whose sums come to more than the partial-sum buffer holds
    (28014, 4992, 32, False),   # tall and many columns: two launches of sixteen
    (28014, 4992, 31, False),   # sixteen and fifteen
    (6704, 9728, 10, True),     # fp32 tokens: more than 200 KB of shared memory, one batch
    (9001, 11008, 7, True),
])
def test_exact_tall(rows, k, m, f32):
    test_exact(rows, k, m, f32)


@pytest.mark.parametrize("rows,k,m,f32", [
    (16, 32, 17, False), (3001, 2016, 24, False),            # one slice
    (260, 2080, 20, False), (7000, 3104, 23, False),         # clusters; several batches
    (30, 65536, 24, False),                                  # memory
    (100, 3200, 6, True), (3001, 4128, 8, True), (2000, 96, 7, True),
])
def test_exact_three_groups_of_columns(rows, k, m, f32):
    test_exact(rows, k, m, f32)
