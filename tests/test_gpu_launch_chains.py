"""Kernels that are placed before the one in front of them has finished, and rows that steer a kernel's scale.

The fp32 operations and the prefill kernels are launched with programmatic stream serialization: a call must see all that the
calls before it wrote, also where it rewrites what they still read.  Bounds are stated beside the comparisons."""
import pytest

torch = pytest.importorskip("torch")

from warpforge_b200 import _native as N, quant as Q  # noqa: E402
from warpforge_b200.backend import CudaContext, QuantizedWeight  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return CudaContext(0)


@pytest.mark.parametrize("rows,n", [(1, 512), (3, 513), (300, 2000), (700, 4096), (64, 16388)])
def test_fp32_operations_in_a_chain(ctx, rows, n):
    """h <- h + swiglu(rms_norm(h), softmax(h)), forty times without a pause, every buffer reused."""
    lib, hd, ck = ctx._lib, ctx.handle, ctx._ck
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    h = torch.randn(rows, n, device="cuda", generator=g)
    gamma = 1 + 0.1 * torch.randn(n, device="cuda", generator=g)
    a, b, c = (torch.empty_like(h) for _ in range(3))
    ref = h.double()
    torch.cuda.synchronize()
    p = lambda t: t.data_ptr()  # noqa: E731
    for _ in range(40):
        ck("rms", lib.wf_rms_norm(hd, p(h), p(gamma), p(a), rows, n, 1e-5, 0))
        ck("softmax", lib.wf_softmax(hd, p(h), p(b), rows, n, 0))
        ck("swiglu", lib.wf_swiglu(hd, p(a), p(b), p(c), rows * n, 0))
        ck("add", lib.wf_add(hd, p(h), p(c), p(h), rows * n, 0))
        r = ref / torch.sqrt((ref * ref).mean(-1, keepdim=True) + 1e-5) * gamma.double()
        ref = ref + r * torch.sigmoid(r) * torch.softmax(ref, -1)
    ctx.synchronize()
    # forty steps of about eight fp32 roundings each: 320 * 2^-24 = 2e-5 of the largest value
    assert (h.double() - ref).abs().max() <= 4e-5 * ref.abs().max()


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
    assert not torch.isfinite(outs[1][7]).any()
    assert not torch.isfinite(outs[1][5]).all()
    ref = clean.double() @ torch.from_numpy(w.dequantize_to_array()).cuda().double().T
    # every weight rounded once to fp16 (2^-12 of it, evenly spread): 3e-4 of a row's root mean square
    err = (outs[0].double() - ref).pow(2).mean(1).sqrt()
    assert (err <= 3e-4 * ref.pow(2).mean(1).sqrt() + 1e-300).all()
    w.close()


@pytest.mark.parametrize("m", [64, 96])
def test_calls_of_other_shapes_back_to_back(ctx, m):
    """The next call's conversion waits beside the running kernel and rewrites the same scratch: alternating shapes, the same bits."""
    qt = Q.QuantizationType.Q8_0
    shapes = [(5003, 1024), (640, 4096), (2048, 2784)]
    ws = [QuantizedWeight(ctx, qt, Q.synth_weight(qt, r, k, i), r, k) for i, (r, k) in enumerate(shapes)]
    g = torch.Generator(device="cuda").manual_seed(m)
    xs = [torch.randn(m, k, device="cuda", generator=g).bfloat16() for _, k in shapes]
    call = lambda i, y: N.check("q", ctx._lib.wf_qlinear(ctx.handle, ws[i].handle, xs[i].data_ptr(), N.WF_DTYPE_BF16, 1, m, y.data_ptr(), 1, 0), ctx.handle)  # noqa: E731
    alone = []
    for i, (r, _) in enumerate(shapes):
        y = torch.empty(m, r, device="cuda")
        torch.cuda.synchronize()
        call(i, y)
        ctx.synchronize()
        alone.append(y)
    outs = [[torch.empty(m, r, device="cuda") for r, _ in shapes] for _ in range(20)]
    torch.cuda.synchronize()
    for o in outs:
        for i in range(3):
            call(i, o[i])
    ctx.synchronize()
    for o in outs:
        for i in range(3):
            assert torch.equal(o[i], alone[i])
    for w in ws:
        w.close()
