"""Kernels that are placed before the one in front of them has finished, and rows that steer a kernel's scale.

The fp32 operations and the prefill kernels are launched with programmatic stream serialization: a call must see all that the
calls before it wrote, also where it rewrites what they still read.  All kernels are deterministic, so a chain that is issued without a
pause, or replayed from a graph, has the bits of one that is waited for after every call; every step has inputs of its own, so that
whatever is read too early shows."""
import pytest

torch = pytest.importorskip("torch")

from warpforge_b200 import _native as N, quant as Q  # noqa: E402
from warpforge_b200.backend import CudaContext, QuantizedWeight  # noqa: E402

pytestmark = pytest.mark.gpu
STEPS = 12


@pytest.fixture(scope="module")
def ctx():
    return CudaContext(0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _three_ways(ctx, issue, outs):
    """issue(pause): all steps, pause() after every call.  Its outputs: waited for, back to back, replayed."""
    seen = []
    for way in ("waited", "back to back", "graph", "graph again"):
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        if way == "waited":
            issue(ctx.synchronize)
        elif way == "back to back":
            issue(lambda: None)
        else:
            if way == "graph":
                ctx.graph_begin()
                issue(lambda: None)
                graph = ctx.graph_end()
            ctx.graph_launch(graph)
        ctx.synchronize()
        seen.append([o.clone() for o in outs])
    ctx.graph_destroy(graph)
    assert all(torch.isfinite(o).all() for o in seen[0])
    for other in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(seen[0], other))


@pytest.mark.parametrize("rows,n", [(1, 512), (3, 513), (300, 2000), (700, 4096), (64, 16388), (2500, 300)])
def test_fp32_operations_in_a_chain(ctx, rows, n):
    """All operations, each reading what the one before it wrote, scratch buffers rewritten in every step."""
    lib, hd, ck = ctx._lib, ctx.handle, ctx._ck
    g = _gen(rows + n)
    table = torch.randn(1000, n, device="cuda", generator=g)
    idx = torch.randint(0, 1000, (STEPS, rows), device="cuda", generator=g)
    up = torch.randn(STEPS, rows, n, device="cuda", generator=g) * torch.arange(1, STEPS + 1, device="cuda")[:, None, None]
    gamma = 1 + 0.1 * torch.randn(STEPS, n, device="cuda", generator=g)
    beta = 0.1 * torch.randn(STEPS, n, device="cuda", generator=g)
    a, b, c, d = (torch.empty(rows, n, device="cuda") for _ in range(4))
    outs = [torch.empty(rows, n, device="cuda") for _ in range(STEPS)]
    p = lambda t: t.data_ptr()  # noqa: E731

    def issue(pause):
        call = lambda name, *args: (ck(name, getattr(lib, "wf_" + name)(hd, *args, 0)), pause())  # noqa: E731
        for s in range(STEPS):
            call("embedding", p(idx[s]), p(table), p(a), rows, 1000, n)
            if s:
                call("add", p(a), p(outs[s - 1]), p(a), rows * n)
            call("rms_norm", p(a), p(gamma[s]), p(b), rows, n, 1e-5)
            call("swiglu", p(b), p(up[s]), p(c), rows * n)
            call("layer_norm", p(c), p(gamma[s]), p(beta[s]), p(d), rows, n, 1e-5)
            call("gelu", p(d), p(b), rows * n)
            call("softmax", p(b), p(c), rows, n)
            call("silu", p(d), p(a), rows * n)
            call("add", p(a), p(c), p(a), rows * n)
            call("rms_norm", p(a), 0, p(outs[s]), rows, n, 1e-5)

    _three_ways(ctx, issue, outs)


@pytest.mark.parametrize("qname", ["Q4_0", "Q4_K"])
@pytest.mark.parametrize("m", [1, 4, 12, 77, 200])
def test_projections_between_fp32_operations(ctx, qname, m):
    """embedding - rms_norm - projection - add, fp32 tokens: the one-token, the several-token and the tensor-core kernels."""
    lib, hd, ck, k = ctx._lib, ctx.handle, ctx._ck, 1024
    qt = Q.QuantizationType[qname]
    ws = [QuantizedWeight(ctx, qt, Q.synth_weight(qt, k, k, i), k, k) for i in range(2)]
    g = _gen(m)
    table = torch.randn(1000, k, device="cuda", generator=g)
    idx = torch.randint(0, 1000, (STEPS, m), device="cuda", generator=g)
    gamma = 1 + 0.1 * torch.randn(STEPS, k, device="cuda", generator=g)
    a, b, y = (torch.empty(m, k, device="cuda") for _ in range(3))
    outs = [torch.empty(m, k, device="cuda") for _ in range(STEPS)]
    p = lambda t: t.data_ptr()  # noqa: E731

    def issue(pause):
        call = lambda name, *args: (ck(name, getattr(lib, "wf_" + name)(hd, *args, 0)), pause())  # noqa: E731
        for s in range(STEPS):
            call("embedding", p(idx[s]), p(table), p(a), m, 1000, k)
            if s:
                call("add", p(a), p(outs[s - 1]), p(a), m * k)
            call("rms_norm", p(a), p(gamma[s]), p(b), m, k, 1e-5)
            for w in ws:
                ck("q", lib.wf_qlinear(hd, w.handle, p(b), N.WF_DTYPE_F32, 1, m, p(y), 1, 0))
                pause()
                call("rms_norm", p(y), 0, p(b), m, k, 1e-5)
            call("add", p(a), p(b), p(outs[s]), m * k)

    _three_ways(ctx, issue, outs)
    for w in ws:
        w.close()


@pytest.mark.parametrize("m,k", [(33, 1024), (77, 2784), (130, 4096), (300, 5024)])
def test_rows_with_inf_and_nan_keep_to_themselves(ctx, m, k):
    """A bf16 row's scale is its largest finite magnitude; an Inf or a NaN shows in its own row's results only."""
    rows = 272
    qt = Q.QuantizationType.Q4_0
    blocks = Q.synth_weight(qt, rows, k, 5)
    w = QuantizedWeight(ctx, qt, blocks, rows, k)
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    x[1] *= 2.0 ** 100
    x[2] *= 2.0 ** -100
    x[3] = 0
    clean = x.clone()
    x[5, k - 1] = float("inf")
    x[7, 0] = float("nan")
    outs = []
    for t in (clean, x):
        y = torch.empty(m, rows, device="cuda")
        torch.cuda.synchronize()
        N.check("q", ctx._lib.wf_qlinear(ctx.handle, w.handle, t.data_ptr(), N.WF_DTYPE_BF16, 1, m, y.data_ptr(), 1, 0), ctx.handle)
        ctx.synchronize()
        outs.append(y)
    keep = [i for i in range(m) if i not in (5, 7)]
    assert torch.equal(outs[0][keep], outs[1][keep])
    wf = torch.from_numpy(w.dequantize_to_array()).cuda()
    assert torch.isnan(outs[1][7]).all()
    want = wf[:, k - 1] * float("inf")  # NaN where the weight is zero
    assert torch.equal(outs[1][5].nan_to_num(nan=0.0), want.nan_to_num(nan=0.0)) and torch.equal(outs[1][5].isnan(), want.isnan())
    ref = clean.double() @ wf.double().T
    # every weight rounded once to fp16 (2^-12 of it, evenly spread): 3e-4 of a row's root mean square
    err = (outs[0].double() - ref).pow(2).mean(1).sqrt()
    assert (err <= 3e-4 * ref.pow(2).mean(1).sqrt() + 1e-300).all()
    w.close()


# (rows, K, tokens) of the calls in turn: clusters on one token count, and clusters before and behind pairs (300 tokens of
# [4096 x 8224]), whose conversions differ
@pytest.mark.parametrize("shapes", [[(5003, 1024, 64), (640, 4096, 64), (2048, 2784, 64)], [(5003, 1024, 96), (640, 4096, 96), (2048, 2784, 96)],
                                    [(1000, 1024, 64), (4096, 8224, 300), (11008, 1024, 128), (4096, 2048, 512)]])
def test_calls_of_other_shapes_back_to_back(ctx, shapes):
    """The next call's conversion waits beside the running kernel and rewrites the same scratch: alternating shapes, the same bits."""
    qt = Q.QuantizationType.Q8_0
    ws = [QuantizedWeight(ctx, qt, Q.synth_weight(qt, r, k, i), r, k) for i, (r, k, _) in enumerate(shapes)]
    g = _gen(len(shapes))
    xs = [[torch.randn(m, k, device="cuda", generator=g).bfloat16() * (s + 1) for _, k, m in shapes] for s in range(STEPS)]
    outs = [[torch.empty(m, r, device="cuda") for r, _, m in shapes] for _ in range(STEPS)]

    def issue(pause):
        for x, o in zip(xs, outs):
            for w, a, y, (_, _, m) in zip(ws, x, o, shapes):
                ctx._ck("q", ctx._lib.wf_qlinear(ctx.handle, w.handle, a.data_ptr(), N.WF_DTYPE_BF16, 1, m, y.data_ptr(), 1, 0))
                pause()

    _three_ways(ctx, issue, [y for o in outs for y in o])
    for w in ws:
        w.close()
