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
