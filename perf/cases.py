"""Workloads of the quantized-linear path: what a program that serves a GGUF model through this framework has it do.

`listed()` names twelve of them, `draw(rng)` makes more of the same ranges.  A case is one of these kinds:

  program  a decode step's projections as one persistent kernel (ProjectionStack.build_program / run_program),
           1 - 8 tokens
  fused    a decode step with rms_norm, silu * up and the residual adds inside the kernel (FusedDecoderStack.run)
  linear   one projection shape, `copies` distinct weights, one wf_qlinear per weight on device buffers
  layer    the seven projections of a decoder layer, one wf_qlinear each; `world` > 1: one rank's row shard of each
  host     Backend.execute(dot_general) on a host tensor: the form in which the reference's backend is called
  glue     the fp32 operations between the projections of a layer, standalone
  load     a weight from GGUF blocks in host memory to its first answer, and released again

Weights follow the distributions of the benchmark configurations (uniform codes, |N(0,1)| scales), activations are
N(0,1).  Weight copies add up to more than the L2 holds wherever a model's weights would.
"""
from __future__ import annotations

import numpy as np
import torch

from warpforge_b200 import _native as N
from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS, NvidiaBackend, QuantizedWeight, Tensor
from warpforge_b200.decode import FusedDecoderStack, ProjectionStack, StackSpec
from warpforge_b200.quant import QuantizationType

QTYPES = ("Q4_0", "Q4_1", "Q5_0", "Q8_0", "Q4_K")
COPY_BYTES = 150 << 20  # weights one pass of a decode case walks: more than the 126 MB of L2
MAX_COPIES = 48
MAX_FLOPS = 8.0e11      # of a drawn case; the largest listed one has 8.3e11


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # One token of the 7B-shape Q4_0 model: the headline decode step, 224 projections, 3.6 GB of weights.
        dict(name="decode_7b_q4_0", kind="program", qtype="Q4_0", d=4096, ffn=11008, layers=32, m=1),
        # Four sequences decoded together through the several-token program, 8-bit weights.
        dict(name="decode_4tok_q8_0", kind="program", qtype="Q8_0", d=4096, ffn=11008, layers=3, m=4),
        # A decode step with its real data flow, fp32 activations from projection to projection.
        dict(name="decode_fused_q4_k", kind="fused", qtype="Q4_K", d=4096, ffn=11008, layers=4),
        # One op per call, one token: a graph executor that issues the projections one by one.
        dict(name="op_1tok_q4_0", kind="linear", qtype="Q4_0", rows=4096, k=11008, copies=6, m=1, x="bf16"),
        # A batch of sixteen on one rank's row shard of the 70B-shape layer.
        dict(name="shard_16tok_q4_k", kind="layer", qtype="Q4_K", d=8192, kv=1024, ffn=28672, world=8, layers=3, m=16),
        # Prefill of a 512-token prompt, one projection.
        dict(name="prefill_512_q4_k", kind="linear", qtype="Q4_K", rows=14336, k=4096, copies=1, m=512, x="bf16"),
        # Prefill of a long prompt through every projection of a 7B-shape layer.
        dict(name="prefill_2048_q4_0", kind="layer", qtype="Q4_0", d=4096, kv=4096, ffn=11008, world=1, layers=1, m=2048),
        # A short prompt on a small model whose row count and token count fit no tile.
        dict(name="prefill_77_q5_0_ragged", kind="linear", qtype="Q5_0", rows=5003, k=2784, copies=8, m=77, x="bf16"),
        # A prompt whose activations are fp32, the only tensor type the reference's CPU backend has.
        dict(name="prefill_96_f32_q4_1", kind="linear", qtype="Q4_1", rows=11008, k=4096, copies=2, m=96, x="f32"),
        # The smallest call: one fp32 row in host memory in, one out.
        dict(name="host_1tok_q8_0", kind="host", qtype="Q8_0", rows=4096, k=4096, m=1, x="f32"),
        # The fp32 operations of a layer over a long prompt.
        dict(name="glue_2048", kind="glue", family="llama", tokens=2048, d=4096, ffn=11008, heads=8, ctx=2048),
        # Loading a model, tensor by tensor.
        dict(name="load_q4_0", kind="load", qtype="Q4_0", rows=28672, k=4096),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _k(rng, qtype, lo, hi):
    """A K between lo and hi: a multiple of the format's block."""
    b = QuantizationType[qtype].block_size()
    return max(b, int(_log(rng, lo, hi)) // b * b)


def _rows(rng, lo, hi):
    """Row counts of models are multiples of 16 or more; a third of the drawn ones are not."""
    r = int(_log(rng, lo, hi))
    return r if rng.random() < 1 / 3 else max(16, r // 16 * 16)


def _copies(qtype, rows, k):
    return max(1, min(MAX_COPIES, COPY_BYTES // (rows * QuantizationType[qtype].row_bytes(k))))


def draw(rng):
    kind = rng.choice(("program", "fused", "op", "shard", "prefill", "prefill", "prefill_layer", "prefill_f32", "host", "glue", "load"))
    qtype = rng.choice(QTYPES)
    if kind in ("program", "fused"):
        d = _k(rng, qtype, 1024, 4096)
        ffn = _k(rng, qtype, 2.3 * d, 2.8 * d)
        if kind == "fused":
            return dict(kind="fused", qtype=qtype, d=d, ffn=ffn, layers=rng.randint(1, 4))
        m = rng.choice((1, 1, 2, rng.randint(3, 8)))
        m = max(1, min(m, 46000 // ffn))  # the tokens' activations of the widest projection lie in one SM's shared memory
        return dict(kind="program", qtype=qtype, d=d, ffn=ffn, layers=rng.randint(2, 8), m=m)
    if kind == "op":
        rows, k = _rows(rng, 256, 32000), _k(rng, qtype, 1024, 11008)
        x = rng.choice(("bf16", "bf16", "f32"))
        m = rng.choice((1, rng.randint(2, 8), rng.randint(9, 32))) if x == "bf16" else rng.choice((1, rng.randint(2, 10)))
        return dict(kind="linear", qtype=qtype, rows=rows, k=k, copies=_copies(qtype, rows, k), m=m, x=x)
    if kind == "shard":
        d = _k(rng, "Q4_K", 2048, 8192)
        return dict(kind="layer", qtype=rng.choice(("Q4_K", "Q4_0", "Q8_0")), d=d, kv=d // 8, ffn=_k(rng, "Q4_K", 2.6 * d, 3.5 * d),
                    world=rng.choice((2, 4, 8)), layers=rng.randint(2, 4), m=rng.randint(2, 32))
    if kind == "prefill":
        rows, k = _rows(rng, 512, 16384), _k(rng, qtype, 1024, 8192)
        m = int(min(_log(rng, 33, 2048), MAX_FLOPS / 2 / rows / k))
        return dict(kind="linear", qtype=qtype, rows=rows, k=k, copies=1, m=m, x="bf16")
    if kind == "prefill_layer":
        d = _k(rng, qtype, 1024, 4096)
        ffn = _k(rng, qtype, 2.3 * d, 2.8 * d)
        m = int(min(_log(rng, 128, 2048), MAX_FLOPS / 2 / (4 * d * d + 3 * d * ffn)))
        return dict(kind="layer", qtype=qtype, d=d, kv=d, ffn=ffn, world=1, layers=1, m=m)
    if kind == "prefill_f32":
        rows, k = _rows(rng, 512, 11008), _k(rng, qtype, 1024, 8192)
        return dict(kind="linear", qtype=qtype, rows=rows, k=k, copies=1, m=int(_log(rng, 11, 256)), x="f32")
    if kind == "host":
        rows, k = _rows(rng, 256, 11008), _k(rng, qtype, 512, 8192)
        return dict(kind="host", qtype=qtype, rows=rows, k=k, m=rng.choice((1, 1, rng.randint(2, 32))), x=rng.choice(("f32", "bf16")))
    if kind == "glue":
        d = int(_log(rng, 512, 8192)) // 4 * 4
        return dict(kind="glue", family=rng.choice(("llama", "gpt")), tokens=int(_log(rng, 1, 2048)), d=d,
                    ffn=int(rng.uniform(2.3, 4) * d), heads=8, ctx=int(_log(rng, 16, 4096)))
    rows, k = _rows(rng, 1024, 28672), _k(rng, qtype, 1024, 4096)
    return dict(kind="load", qtype=qtype, rows=rows, k=k)


# ------------------------------------------------------------------------------------------------ inputs
_backend = None


def backend() -> NvidiaBackend:
    """A program has one backend (one context, one stream) for its lifetime."""
    global _backend
    if _backend is None:
        _backend = NvidiaBackend(0)
    return _backend


def _fp16_scales(gen, nb, s):
    return (torch.randn(nb, device="cuda", generator=gen).abs() * s).half().view(torch.uint8).view(nb, 2)


def blocks_of(qtype: str, rows: int, k: int, gen) -> np.ndarray:
    """GGUF blocks [rows, row bytes] in host memory."""
    qt = QuantizationType[qtype]
    nb, size = rows * (k // qt.block_size()), qt.bytes_per_block()
    t = torch.randint(0, 256, (nb, size), dtype=torch.uint8, device="cuda", generator=gen)
    t[:, 0:2] = _fp16_scales(gen, nb, 0.01 if qtype == "Q4_K" else 0.02)
    if qtype == "Q4_1":
        t[:, 2:4] = (-8 * (torch.randn(nb, device="cuda", generator=gen).abs() * 0.02)).half().view(torch.uint8).view(nb, 2)
    elif qtype == "Q4_K":
        t[:, 2:4] = _fp16_scales(gen, nb, 0.01)
    elif qtype == "Q8_0":
        c = t[:, 2:]
        c[c == 0x80] = 0x81  # codes in [-127, 127]
    return t.view(rows, -1).cpu().numpy()


class _Held:
    """Handles and buffers of the framework, given back with the last thing that refers to them."""

    def __init__(self, *closers):
        self.closers = closers

    def __del__(self):
        for c in self.closers:
            c()


class _DeviceRow:
    """A buffer of the framework's context, readable by torch."""

    def __init__(self, ptr, shape, held):
        self.held = held
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f4", "version": 3}


def _view(held, ptr, *shape):
    return torch.as_tensor(_DeviceRow(ptr, shape, held), device="cuda")


class State:
    """What a program keeps between calls."""

    def __init__(self, run, held=None, keep=None):
        self.run, self.held, self.keep = run, held, keep


def _projections(c):
    """(rows of this rank's shard, k) of a layer's seven projections."""
    d, kv, ffn, w = c["d"], c["kv"], c["ffn"], c["world"]
    return [(r // w, k) for r, k in ((d, d), (kv, d), (kv, d), (d, d), (ffn, d), (ffn, d), (d, ffn))]


def _calls(c):
    """(rows, k) of every wf_qlinear of a pass."""
    return [(c["rows"], c["k"])] * c["copies"] if c["kind"] == "linear" else _projections(c) * c["layers"]


def _activations(m, k, x, gen):
    a = torch.randn(m, k, device="cuda", generator=gen)
    return a.bfloat16() if x == "bf16" else a


def _prepare_calls(c, gen):
    ctx = backend().cuda_context
    x = c.get("x", "bf16")
    dtype = N.WF_DTYPE_BF16 if x == "bf16" else N.WF_DTYPE_F32
    xs, calls, outs, made, weights = {}, [], [], {}, []
    for rows, k in _calls(c):
        if k not in xs:
            xs[k] = _activations(c["m"], k, x, gen)
        if c["kind"] == "layer" or (rows, k) not in made:
            made[rows, k] = blocks_of(c["qtype"], rows, k, gen)
        w = QuantizedWeight(ctx, QuantizationType[c["qtype"]], made[rows, k], rows, k)
        y = torch.empty(c["m"], rows, device="cuda")
        calls.append((w.handle, xs[k].data_ptr(), y.data_ptr()))
        outs.append(y)
        weights.append(w)
    lib, h, m = ctx._lib, ctx.handle, c["m"]

    def run():
        for w, xp, yp in calls:
            rc = lib.wf_qlinear(h, w, xp, dtype, 1, m, yp, 1, 0)
            if rc:
                N.check("wf_qlinear", rc, h)
        return outs

    return State(run, _Held(*[w.close for w in weights]), xs)


def _prepare_program(c, seed):
    ctx = backend().cuda_context
    d, ffn = c["d"], c["ffn"]
    spec = StackSpec("stack", QuantizationType[c["qtype"]], c["layers"], (
        ("wq", d, d), ("wk", d, d), ("wv", d, d), ("wo", d, d), ("wgate", ffn, d), ("wup", ffn, d), ("wdown", d, ffn)), 1000 + seed)
    st = ProjectionStack(ctx, spec, tokens=c["m"])
    st.build_program()
    held = _Held(st.close, *[lambda p=p: ctx.free(p) for p in list(st.x_dev.values()) + list(st.y_dev.values())])
    outs = [_view(held, st.y_dev[n], c["m"], r) for n, r, _ in spec.projections]

    def run():
        st.run_program()
        return outs

    return State(run, held)


def _prepare_fused(c, seed):
    ctx = backend().cuda_context
    st = FusedDecoderStack(ctx, QuantizationType[c["qtype"]], c["d"], c["ffn"], c["layers"], seed=1000 + seed)
    names = ["%s_%d" % (n, l) for l in range(c["layers"]) for n in ("q", "k", "v", "hmid", "gate", "up")] + ["h%d" % (l + 1) for l in range(c["layers"])]
    held = _Held(st.close)
    outs = [_view(held, st.dev[n], st.host[n].size) for n in names]

    def run():
        st.run()
        return outs

    return State(run, held)


def _prepare_host(c, gen):
    be = backend()
    w = QuantizedWeight(be.cuda_context, QuantizationType[c["qtype"]], blocks_of(c["qtype"], c["rows"], c["k"], gen), c["rows"], c["k"])
    a = _activations(c["m"], c["k"], c["x"], gen).cpu()
    x = Tensor(a.numpy(), "f32") if c["x"] == "f32" else Tensor(a.view(torch.int16).numpy().view(np.uint16), "bf16")
    op = DotGeneralOp(LINEAR_DIMS, (c["m"], c["rows"]))
    return State(lambda: be.execute(op, [x, w])[0].data, _Held(w.close))


def _prepare_load(c, gen):
    ctx = backend().cuda_context
    qt, rows, k = QuantizationType[c["qtype"]], c["rows"], c["k"]
    blocks = blocks_of(c["qtype"], rows, k, gen)
    x, y = _activations(1, k, "bf16", gen), torch.empty(1, rows, device="cuda")
    lib, h = ctx._lib, ctx.handle

    def run():
        w = QuantizedWeight(ctx, qt, blocks, rows, k)
        N.check("wf_qlinear", lib.wf_qlinear(h, w.handle, x.data_ptr(), N.WF_DTYPE_BF16, 1, 1, y.data_ptr(), 1, 0), h)
        w.close()
        return y

    return State(run)


def _prepare_glue(c, gen):
    ctx = backend().cuda_context
    lib, h = ctx._lib, ctx.handle
    t, d, ffn, srows, n = c["tokens"], c["d"], c["ffn"], c["tokens"] * c["heads"], c["ctx"]
    new = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    vocab = 32000
    table = new(vocab, d)
    idx = torch.randint(0, vocab, (t,), device="cuda", generator=gen)
    gamma, beta, proj, scores = 1 + 0.1 * new(d), 0.1 * new(d), new(t, d), new(srows, n)
    gate, up = new(t, ffn), new(t, ffn)
    emb, normed, probs, act, res = (torch.empty_like(v) for v in (proj, proj, scores, gate, proj))
    p = {k: v.data_ptr() for k, v in dict(table=table, idx=idx, gamma=gamma, beta=beta, proj=proj, scores=scores, gate=gate, up=up,
                                          emb=emb, normed=normed, probs=probs, act=act, res=res).items()}
    llama = c["family"] == "llama"
    ck = ctx._ck

    def run():
        ck("wf_embedding", lib.wf_embedding(h, p["idx"], p["table"], p["emb"], t, vocab, d, 0))
        if llama:
            ck("wf_rms_norm", lib.wf_rms_norm(h, p["emb"], p["gamma"], p["normed"], t, d, 1e-5, 0))
        else:
            ck("wf_layer_norm", lib.wf_layer_norm(h, p["emb"], p["gamma"], p["beta"], p["normed"], t, d, 1e-5, 0))
        ck("wf_softmax", lib.wf_softmax(h, p["scores"], p["probs"], srows, n, 0))
        ck("wf_add", lib.wf_add(h, p["emb"], p["proj"], p["res"], t * d, 0))
        if llama:
            ck("wf_swiglu", lib.wf_swiglu(h, p["gate"], p["up"], p["act"], t * ffn, 0))
        else:
            ck("wf_gelu", lib.wf_gelu(h, p["gate"], p["act"], t * ffn, 0))
        return [emb, normed, probs, res, act]

    return State(run, keep=(table, idx, gamma, beta, proj, scores, gate, up))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "program":
        return _prepare_program(case, seed)
    if kind == "fused":
        return _prepare_fused(case, seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return {"linear": _prepare_calls, "layer": _prepare_calls, "host": _prepare_host, "glue": _prepare_glue, "load": _prepare_load}[kind](case, gen)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    c, kind = case, case["kind"]
    if kind == "glue":
        t, d, ffn, n = c["tokens"], c["d"], c["ffn"], c["tokens"] * c["heads"] * c["ctx"]
        # embedding, norm and add on [t, d]; softmax; swiglu reads two tensors, gelu one
        floats = (2 + 2 + 3) * t * d + 2 * n + (3 if c["family"] == "llama" else 2) * t * ffn
        return {"bytes": 4 * floats + 8 * t, "flops": 0}
    qt = QuantizationType[c["qtype"]]
    if kind in ("program", "fused"):
        d, ffn, m = c["d"], c["ffn"], c.get("m", 1)
        weights = c["layers"] * (4 * d * qt.row_bytes(d) + 2 * ffn * qt.row_bytes(d) + d * qt.row_bytes(ffn))
        macs = m * c["layers"] * (4 * d * d + 3 * d * ffn)
        if kind == "program":  # bf16 rows in (one per input of a projection group), fp32 rows out
            rows = m * c["layers"] * (2 * (3 * d + ffn) + 4 * (5 * d + 2 * ffn))
        else:  # the residual stream and attention's rows in, q, k, v, gate, up and the new streams out
            rows = c["layers"] * 4 * (3 * d + 2 * ffn + 4 * d)
        return {"bytes": weights + rows, "flops": 2 * macs}
    calls = _calls(c) if kind in ("linear", "layer") else [(c["rows"], c["k"])]
    m, xb = c.get("m", 1), 4 if c.get("x") == "f32" else 2
    total = sum(r * qt.row_bytes(k) + m * k * xb + m * r * 4 for r, k in calls)
    if kind == "load":  # the blocks cross to the device, are written there and read once by the projection
        total += 2 * c["rows"] * qt.row_bytes(c["k"])
    return {"bytes": total, "flops": sum(2 * m * r * k for r, k in calls)}


def tolerance(case):
    """fp32 sums of exact products everywhere but in the many-token tensor-core path, which rounds every dequantized
    weight once to fp16 (2^-12, uniformly distributed: about 1.2e-4 of the result for one implementation)."""
    if case["kind"] in ("linear", "layer") and case["m"] > 32 and case.get("x", "bf16") == "bf16":
        return {"rel": 4e-4}
    if case["kind"] == "fused":  # several layers of fp32 sums, each fed by the one before
        return {"rel": 3e-5}
    return {"rel": 1e-5}
