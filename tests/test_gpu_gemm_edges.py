"""The tensor-core kernels at the edges of their tiles: K-splitting clusters (128 rows x up to 128 tokens; ranks with no tokens of their own to finish, several tiles
per cluster, clusters of one), CTA pairs (256 rows x up to 256 tokens, cut tiles, whole tiles first), K that ends inside a span of 64, and fp32 tokens.  Where a
test is about one of the kernels it asks wf_plan_many_tokens, which answers for a device of 148 SMs, whether that is the one that runs.

bf16 tokens: the bars of test_gpu_gemm.py.  fp32 tokens: products are exact to 2^-22 and an accumulator takes at most 32
steps between two drains, each cutting the partial sum off at its 24th bit: 32 x 2^-23 = 3.8e-6 of the result at
the very most, in the 2-norm against float64."""
import collections
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from warpforge_b200 import quant as Q

pytestmark = pytest.mark.gpu

QT = {"q4_0": O.Q4_0, "q4_1": O.Q4_1, "q5_0": O.Q5_0, "q8_0": O.Q8_0, "q4_k": O.Q4_K}


@pytest.fixture(scope="module")
def backend():
    from warpforge_b200.backend import NvidiaBackend

    b = NvidiaBackend(0)
    yield b
    b.close()


def _run(backend, oracle, name, rows, k, x, tensor):
    """Two calls (the second finds the scratch of the first) and the exact product."""
    from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS

    qt = Q.QuantizationType[name.upper()]
    blocks = Q.synth_weight(qt, rows, k, rows + k + len(x))
    w = backend.upload_weight(qt, blocks, rows, k)
    got = [backend.execute(DotGeneralOp(LINEAR_DIMS, (len(x), rows)), [tensor, w])[0].data for _ in range(2)]
    w.close()
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    wf = oracle.dequant(QT[name], blocks, rows * k).reshape(rows, k).astype(np.float64)
    return got[0], x.astype(np.float64) @ wf.T


Plan = collections.namedtuple("Plan", "pairs tokens ctas groups waves")


def _plan(backend, name, rows, k, m, f32=False):
    ctx = backend.cuda_context
    v = [ctypes.c_int() for _ in Plan._fields]
    ctx._ck("plan", ctx._lib.wf_plan_many_tokens(ctx.handle, Q.QuantizationType[name.upper()].ggml_type, rows, k, m, int(f32), *map(ctypes.byref, v)))
    return Plan(*(x.value for x in v))


def _run_sampled(backend, oracle, name, rows, k, x, tensor):
    """As _run for a large weight: three rows of every 128 (the first, the last, one between), all tokens."""
    from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS

    qt = Q.QuantizationType[name.upper()]
    blocks = Q.synth_weight(qt, rows, k, rows + k + len(x))
    w = backend.upload_weight(qt, blocks, rows, k)
    got = [backend.execute(DotGeneralOp(LINEAR_DIMS, (len(x), rows)), [tensor, w])[0].data for _ in range(2)]
    w.close()
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    sample = np.unique(np.concatenate([np.arange(0, rows, 128), np.minimum(np.arange(127, rows + 127, 128), rows - 1), np.arange(rows // 128) * 128 + 61]))
    wf = oracle.dequant(QT[name], blocks[sample], len(sample) * k).reshape(-1, k).astype(np.float64)
    return got[0][:, sample], x.astype(np.float64) @ wf.T


@pytest.mark.parametrize("name", sorted(QT))
@pytest.mark.parametrize("rows,k,m", [
    (130, 352, 33), (1000, 1120, 80), (700, 5152, 77), (2500, 672, 128),  # clusters; K ends inside a span
    (3000, 544, 129), (3072, 1024, 257), (2900, 288, 513), (1600, 2080, 1100),  # clusters of one, on several token tiles of 64 to 128
    (300, 800, 300), (128, 4128, 600),  # few tiles: clusters on several token tiles
    (2900, 4096, 300), (2900, 4128, 129), (2900, 8192, 130), (2900, 8224, 300),  # K at the ends of what the conversion holds of a row
    (5100, 4128, 1000), (3600, 8224, 300),  # either kernel, by a hair
])
def test_bf16_tokens(backend, oracle, name, rows, k, m):
    from warpforge_b200.backend import Tensor

    if name == "q4_k":
        k = max(256, k // 256 * 256)
    xb = Q.synth_activation_bf16(m, k, rows + m)
    got, want = _run(backend, oracle, name, rows, k, Q.bf16_bits_to_float(xb), Tensor.from_bf16_bits(xb))
    d = got - want
    assert np.max(np.abs(d)) <= 1e-3 * np.max(np.abs(want))
    assert np.linalg.norm(d) <= 3e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("name,rows,k,m,tokens,pieces", [(name, *shape) for names, shape in [  # pieces: about how many pairs share a tile
    (("q4_0", "q4_1", "q4_k"), (19000, 6144, 90, 96, 1)),   # rows that the conversion's long form holds
    (sorted(QT), (19000, 6144, 125, 128, 1)),
    (sorted(QT), (6500, 3904, 300, 160, 1)),                # rows that the short form holds
    (("q4_0", "q4_1", "q4_k"), (3096, 8800, 306, 160, 3)),  # more than either holds; few tiles, each cut several times
    (sorted(QT), (4700, 8224, 520, 192, 1)),
    (sorted(QT), (784, 11168, 1319, 224, 3)),
    (sorted(QT), (7100, 3104, 1030, 224, 1)),
    (sorted(QT), (8000, 3104, 1250, 256, 1)),
] for name in names])
def test_pairs_of_ctas(backend, oracle, name, rows, k, m, tokens, pieces):
    """Sizes from which the cost functions take the CTA pairs, ragged in rows, K and tokens."""
    from warpforge_b200.backend import Tensor

    if name == "q4_k":
        k = k // 256 * 256
    p = _plan(backend, name, rows, k, m)
    tiles = -(-rows // 256) * -(-m // tokens)
    assert p.pairs == 1 and p.ctas == 2 and p.tokens == tokens and p.waves == 0
    assert tiles % p.groups and (pieces == 1 or p.groups >= (pieces - 0.3) * tiles)  # tiles are cut
    bits = Q.synth_activation_bf16(m, k, rows + m)
    got, want = _run_sampled(backend, oracle, name, rows, k, Q.bf16_bits_to_float(bits).reshape(m, k), Tensor.from_bf16_bits(bits))
    assert np.max(np.abs(got - want)) <= 1e-3 * np.max(np.abs(want))
    assert np.linalg.norm(got - want) <= 3e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("name,rows,k,m,pairs", [  # us by clusters of one / by pairs
    ("q4_k", 8192, 8192, 256, 1),  # 42.7 / 40.2
    ("q4_1", 9000, 6976, 700, 1),  # 91.8 / 75.7
    ("q8_0", 5003, 2784, 512, 0),  # 25.0 / 28.7
    ("q4_0", 4096, 4096, 512, 0),  # 18.6 / 28
])
def test_choice_of_the_kernel(backend, name, rows, k, m, pairs):
    assert _plan(backend, name, rows, k, m).pairs == pairs


@pytest.mark.parametrize("name,rows,k,m,waves", [  # weights of 37 MB and more, 132 MB read again
    ("q8_0", 6000, 6016, 1200, 1),  # then 29 of 47 units a pair
    ("q5_0", 6000, 6016, 2000, 2),
    ("q4_k", 8100, 7936, 1100, 1),  # the rest is more than a tile a pair
    ("q4_0", 8190, 8224, 1030, 1),
    ("q4_1", 7700, 8000, 1100, 1),
])
def test_pairs_that_take_whole_tiles_first(backend, oracle, name, rows, k, m, waves):
    from warpforge_b200.backend import Tensor

    p = _plan(backend, name, rows, k, m)
    assert p.pairs == 1 and p.waves == waves
    bits = Q.synth_activation_bf16(m, k, rows + m)
    got, want = _run_sampled(backend, oracle, name, rows, k, Q.bf16_bits_to_float(bits).reshape(m, k), Tensor.from_bf16_bits(bits))
    assert np.max(np.abs(got - want)) <= 1e-3 * np.max(np.abs(want))
    assert np.linalg.norm(got - want) <= 3e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("name", sorted(QT))
@pytest.mark.parametrize("rows,k,m,f32", [
    (10300, 6688, 70, False),
    (26453, 2432, 16, True),  # the few rows of fp32 whose GEMM lets the next conversion in early
    (1950, 3648, 200, True),  # several token tiles
    (7600, 1344, 205, True),
])
def test_clusters_that_split_several_tiles(backend, oracle, name, rows, k, m, f32):
    """More than one tile to a cluster of several ranks: the second phases of the exchange's barriers, exchange and sums used again, and (fp32) more
    than one group of four units to a rank, so that the accumulators' turns go on over the tiles."""
    from warpforge_b200.backend import Tensor

    if name == "q4_k":
        k = k // 256 * 256
    p = _plan(backend, name, rows, k, m, f32)
    tiles = -(-rows // 128) * -(-m // p.tokens)
    assert p.pairs == 0 and p.ctas > 1 and tiles > p.groups and k / 128 / p.ctas > 4
    if f32:
        x = Q.synth_activation_f32(m, k, rows + m)
        t = Tensor.from_float_array(x)
    else:
        bits = Q.synth_activation_bf16(m, k, rows + m)
        x, t = Q.bf16_bits_to_float(bits).reshape(m, k), Tensor.from_bf16_bits(bits)
    got, want = _run_sampled(backend, oracle, name, rows, k, x, t)
    assert np.linalg.norm(got - want) <= (3.8e-6 if f32 else 3e-4) * np.linalg.norm(want)
    assert np.max(np.abs(got - want)) <= (3.8e-5 if f32 else 1e-3) * np.max(np.abs(want))  # f32: ten times the 2-norm's bar


@pytest.mark.parametrize("name,f32", [("q4_0", False), ("q8_0", False), ("q4_k", False), ("q4_1", True), ("q8_0", True), ("q4_k", True)])
@pytest.mark.parametrize("rows,k,tokens", [
    (20600, 128, (40,)),  # more tiles than clusters of one unit each: the sets of dequantizing warps take tiles by turns
    (300, 1184, (16, 33, 48, 65, 80, 95)),  # every length of the ring of weights in TMEM; a last tile of the weight that is partly empty
    (2600, 2720, (64, 96, 113)),
])
def test_rings_of_weights_in_tmem(backend, oracle, name, f32, rows, k, tokens):
    from warpforge_b200.backend import Tensor

    if name == "q4_k":
        k = max(256, k // 256 * 256)
    for m in tokens:
        if f32:
            x = Q.synth_activation_f32(m, k, rows + m)
            t = Tensor.from_float_array(x)
        else:
            bits = Q.synth_activation_bf16(m, k, rows + m)
            x, t = Q.bf16_bits_to_float(bits), Tensor.from_bf16_bits(bits)
        got, want = _run(backend, oracle, name, rows, k, x, t)
        assert np.linalg.norm(got - want) <= (3.8e-6 if f32 else 3e-4) * np.linalg.norm(want)
        assert np.max(np.abs(got - want)) <= (3.8e-5 if f32 else 1e-3) * np.max(np.abs(want))  # f32: ten times the 2-norm's bar


@pytest.mark.parametrize("name", sorted(QT))
@pytest.mark.parametrize("rows,k,m", [(100, 96, 11), (257, 2080, 24), (1000, 4000, 96), (640, 1024, 97), (2100, 544, 200)])
def test_fp32_tokens(backend, oracle, name, rows, k, m):
    from warpforge_b200.backend import Tensor

    if name == "q4_k":
        k = max(256, k // 256 * 256)
    x = Q.synth_activation_f32(m, k, rows + m)
    x[1] *= 1e20  # a scale of its own per token
    got, want = _run(backend, oracle, name, rows, k, x, Tensor.from_float_array(x))
    for rows_of in (slice(1, 2), np.r_[0, 2:m]):
        assert np.linalg.norm((got - want)[rows_of]) <= 3.8e-6 * np.linalg.norm(want[rows_of])


def test_fp32_tokens_keep_fp32s_range(backend, oracle):
    """Weights beyond fp16's range (a scale of 20000): the many-token kernel cannot hold them, the call still answers."""
    from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS, Tensor

    rows, k, m = 64, 256, 40
    blocks = Q.synth_q8_0(rows, k, 3).reshape(rows, -1, 34).copy()
    blocks[5, 2, :2] = np.frombuffer(np.float16(20000.0).tobytes(), np.uint8)
    blocks = blocks.reshape(rows, -1)
    x = Q.synth_activation_f32(m, k, 4)
    w = backend.upload_weight(Q.QuantizationType.Q8_0, blocks, rows, k)
    got = backend.execute(DotGeneralOp(LINEAR_DIMS, (m, rows)), [Tensor.from_float_array(x), w])[0].data
    w.close()
    want = x.astype(np.float64) @ oracle.dequant(O.Q8_0, blocks, rows * k).reshape(rows, k).astype(np.float64).T
    assert np.linalg.norm(got - want) <= 3.8e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("f32", [True, False])
def test_rows_of_the_smallest_magnitudes(backend, oracle, f32):
    """Rows whose largest magnitude lies on either side of 2^-112 (where the scale to fp16's range reaches its end), down to
    subnormal floats, next to ordinary ones and a row of zeros.  Weights of magnitude 1e3 .. 1e4 keep y normal, so the bars
    of the other tests hold row by row."""
    from warpforge_b200.backend import DotGeneralOp, LINEAR_DIMS, Tensor

    rows, k, m = 200, 544, 40
    blocks = Q.synth_q8_0(rows, k, 3).reshape(rows, -1, 34).copy()
    blocks[:, :, :2] = np.random.default_rng(1).uniform(100, 400, (rows, k // 32)).astype(np.float16)[..., None].view(np.uint8)
    blocks = blocks.reshape(rows, -1)
    x = Q.synth_activation_f32(m, k, 4)
    small = {1: 2.0 ** -115, 2: 1e-35, 3: 2.0 ** -126, 4: 2.0 ** -132, 5: 0.0, 6: 2.0 ** -111, 7: 2.0 ** -100, 9: 1e30}
    for r, scale in small.items():
        x[r] = (x[r].astype(np.float64) * scale).astype(np.float32)
    if not f32:
        bits = Q.float_to_bf16_bits(x).reshape(m, k)
        x = Q.bf16_bits_to_float(bits).reshape(m, k)
    w = backend.upload_weight(Q.QuantizationType.Q8_0, blocks, rows, k)
    t = Tensor.from_float_array(x) if f32 else Tensor.from_bf16_bits(bits)
    got = backend.execute(DotGeneralOp(LINEAR_DIMS, (m, rows)), [t, w])[0].data
    w.close()
    want = x.astype(np.float64) @ oracle.dequant(O.Q8_0, blocks, rows * k).reshape(rows, k).astype(np.float64).T
    assert np.any(x[4]) and np.max(np.abs(x[4])) < 2.0 ** -126 * 16 and not np.any(got[5])
    for r in range(m):
        assert np.linalg.norm(got[r] - want[r]) <= (3.8e-6 if f32 else 3e-4) * np.linalg.norm(want[r]), r
