"""Raw-row mode where several tiles share the copy of an output row: the CTAs' ranges begin and end inside rows, with one to many tiles,
so that rows with a tile of only one of the two issuing warps occur at either end.  Against the CPU checker bit for bit."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_conv import run_gpu
from tennis_b200 import ops

pytestmark = pytest.mark.gpu

# N, C, H, W, O, K, stride, pad
GEOMETRIES = [
    (1, 3, 30, 250, 16, 3, 1, 1),     # two segments, 60 tiles: one a CTA
    (2, 3, 40, 300, 8, 3, 1, 1),      # three segments, 240 tiles: one or two
    (3, 3, 77, 380, 40, 3, 1, 1),     # three segments, four or five tiles
    (2, 4, 131, 400, 20, 5, 1, 2),    # four segments, seven or eight tiles
    (2, 3, 90, 520, 70, 7, 2, 3),     # strided, pixel stride 16 bytes at half the width; three segments, two channel tiles
    (1, 3, 160, 256, 300, 3, 1, 1),   # two channel tiles: CTAs that replace their weights
]


@pytest.mark.parametrize("geo", GEOMETRIES)
def test_raw_row_segments(checker, geo):
    N, C, H, W, O, K, stride, pad = geo
    plan = ops.ConvPlan((N, C, H, W), (O, C, K, K), (pad,) * 4, (stride,) * 2, (1, 1), raw_row_mode=2)
    assert "mode=rows" in plan.describe()
    rng = np.random.default_rng(5)
    x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-128, 128, (O, C, K, K)).astype(np.int8)
    dq = rng.uniform(1e-4, 1e-3, O).astype(np.float32)
    bias = rng.normal(0, 0.1, O).astype(np.float32)
    rq = [np.float32(2.5)] * N
    y = checker.activation(checker.add_bias(checker.conv2d_quantized(x, w, (pad,) * 4, (stride,) * 2, (1, 1), dq, 0.0), bias), "relu", 0.0)
    for kw in (dict(want_f32=False, rq=rq, i8_layout="nhwc"), dict(), dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc")):
        got = run_gpu(x, w, (pad,) * 4, (stride,) * 2, (1, 1), dq, bias, "relu", 0.0, want_acc=False, tune=dict(raw_row_mode=2), **kw)
        if kw.get("want_f32", True):
            assert same_bits(got["f32"], y)
        if "rq" in kw:
            assert np.array_equal(got["i8"], checker.quantize(y, rq))
