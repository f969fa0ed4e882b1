"""The persistent program kernels (csrc/wf_decode.cu: gemv1_program_kernel, gemv_program_kernel), which programs of several
ranks run on.  On one rank a program takes them only where an op reads a part of what a longer K staged, so every program
here has such an op; that it is ONE launch is checked.  All block formats, one and several tokens, and the fp32 operations
in the staging and the store, against the CPU oracle (a bar of 1e-3 of each buffer's largest magnitude, as in the other
program tests; same bits from run to run)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu

OQ = {"Q4_0": O.Q4_0, "Q4_1": O.Q4_1, "Q8_0": O.Q8_0, "Q4_K": O.Q4_K, "Q5_0": O.Q5_0}


class _Program:
    """Op list -> program; every op's output row(s) in a buffer of its own."""

    def __init__(self, ctx, qt, m):
        self.ctx, self.qt, self.m = ctx, qt, m
        self.w, self.x, self.y, self.flags, self.kind, self.aux, self.eps, self.res, self.rows, self.blocks = ([] for _ in range(10))

    def upload(self, a):
        d = self.ctx.allocate(a.nbytes)
        self.ctx.copy_to_device(d, a)
        return d

    def op(self, rows, k, x, new=True, kind=0, aux=0, eps=0.0, residual=0):
        from warpforge_b200 import _native as N
        from warpforge_b200.backend import QuantizedWeight

        self.blocks.append(Q.synth_weight(self.qt, rows, k, 70 + len(self.w)))
        self.w.append(QuantizedWeight(self.ctx, self.qt, self.blocks[-1], rows, k))
        self.x.append(x)
        self.y.append(self.ctx.allocate(self.m * rows * 4))
        self.flags.append(N.WF_OP_NEW_X | N.WF_OP_DEPENDS if new else 0)
        self.kind.append(kind)
        self.aux.append(aux)
        self.eps.append(eps)
        self.res.append(residual)
        self.rows.append(rows)
        return self.y[-1]

    def run(self):
        """The outputs after each of two runs, and the launches a run took."""
        ctx, lib, n = self.ctx, self.ctx._lib, len(self.w)
        arr = lambda v, t: (t * n)(*v)
        prog = ctypes.c_int64()
        ctx._ck("create", lib.wf_program_create_fused(
            ctx.handle, n, arr([w.handle for w in self.w], ctypes.c_int64), arr(self.x, ctypes.c_int64), arr(self.y, ctypes.c_int64),
            arr(self.flags, ctypes.c_int), arr(self.kind, ctypes.c_int), arr(self.aux, ctypes.c_int64), arr(self.eps, ctypes.c_float),
            arr(self.res, ctypes.c_int64), self.m, 1, 0, None, ctypes.byref(prog)))
        got, before = [], ctx.launch_count()
        for _ in range(2):
            ctx._ck("run", lib.wf_program_run(ctx.handle, prog.value, 0))
            ctx.synchronize()
            got.append([np.empty((self.m, r), np.float32) for r in self.rows])
            for a, p in zip(got[-1], self.y):
                ctx.copy_to_host(a, p)
        launches = ctx.launch_count() - before
        ctx._ck("destroy", lib.wf_program_destroy(ctx.handle, prog.value))
        assert launches == 2, "one persistent launch per run"
        for a, b in zip(*got):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        return got[0]


def _close(got, want):
    assert np.isfinite(got).all() and np.max(np.abs(got - want)) <= 1e-3 * np.max(np.abs(want))


@pytest.mark.parametrize("qname", sorted(OQ))
@pytest.mark.parametrize("m", [1, 2, 5, 8])
def test_projections(oracle, qname, m):
    from warpforge_b200.backend import CudaContext

    ctx = CudaContext(0)
    try:
        p = _Program(ctx, Q.QuantizationType[qname], m)
        xs = {k: Q.synth_activation_bf16(m, k, k) for k in (768, 2560)}
        dev = {k: p.upload(v) for k, v in xs.items()}
        # (rows, k, row of x, new input): joined, a part of the longer input, short, long and ragged row counts
        ops = [(700, 2560, 2560, True), (33, 2560, 2560, False), (2500, 768, 2560, False), (16, 768, 768, True), (5000, 2560, 2560, True), (1, 2560, 2560, False)]
        for rows, k, src, new in ops:
            p.op(rows, k, dev[src], new)
        got = p.run()
        for g, b, (rows, k, src, _) in zip(got, p.blocks, ops):
            x = Q.bf16_bits_to_float(xs[src]).reshape(m, src)[:, :k]
            _close(g, oracle.qlinear(OQ[qname], b, rows, k, np.ascontiguousarray(x), nthreads=oracle.max_threads()).reshape(m, rows))
    finally:
        ctx.close()


@pytest.mark.parametrize("qname", sorted(OQ))
def test_operations_between_projections(oracle, qname):
    """A layer with rms_norm, silu * up and the residual adds inside, and beside q a projection of the first half of the same
    normalised row."""
    from warpforge_b200 import _native as N
    from warpforge_b200.backend import CudaContext

    d, ffn, eps = 1024, 2816, 1e-5
    rng = np.random.default_rng(4)
    h, attn, g1, g2 = (rng.standard_normal(d).astype(np.float32) for _ in range(4))
    g1, g2 = 1 + np.float32(0.1) * g1, 1 + np.float32(0.1) * g2
    ctx = CudaContext(0)
    try:
        p = _Program(ctx, Q.QuantizationType[qname], 1)
        dh, da, dg1, dg2 = (p.upload(a) for a in (h, attn, g1, g2))
        p.op(d, d, dh, True, N.WF_X_RMSNORM_F32, dg1, eps)
        p.op(300, d // 2, dh, False)
        hmid = p.op(d, d, da, True, N.WF_X_F32, residual=dh)
        gate = p.op(ffn, d, hmid, True, N.WF_X_RMSNORM_F32, dg2, eps)
        up = p.op(ffn, d, hmid, False)
        p.op(d, ffn, gate, True, N.WF_X_SWIGLU_F32, up, residual=hmid)
        got = [a.reshape(-1) for a in p.run()]
        lin = lambda i, rows, x: oracle.qlinear(OQ[qname], p.blocks[i], rows, x.size, x.reshape(1, -1), nthreads=oracle.max_threads()).reshape(-1)  # noqa: E731
        x1 = oracle.rms_norm(h.reshape(1, -1), g1, eps).reshape(-1)
        want = [lin(0, d, x1), lin(1, 300, np.ascontiguousarray(x1[:d // 2]))]
        want.append(oracle.add(h, lin(2, d, attn)))
        x2 = oracle.rms_norm(want[2].reshape(1, -1), g2, eps).reshape(-1)
        want += [lin(3, ffn, x2), lin(4, ffn, x2)]
        want.append(oracle.add(want[2], lin(5, d, oracle.swiglu(want[3], want[4]))))
        for g, w in zip(got, want):
            _close(g, w)
    finally:
        ctx.close()
