"""Patch mode over pixel pairs (filters of stride 2 over 17 to 64 channels): odd and even paddings and filter widths, ragged tiles, both
orientations, against the CPU checker bit for bit; an odd width keeps the general path."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_conv import run_gpu
from tennis_b200 import ops

pytestmark = pytest.mark.gpu

# N, C, H, W, O, (KH, KW), padding (top, bottom, left, right)
GEOMETRIES = [
    (1, 64, 32, 16, 64, (3, 3), (1, 1, 1, 1)),       # one tile, exactly
    (2, 32, 33, 34, 85, (3, 3), (1, 1, 1, 1)),       # 17 x 17 pixels: tiles that hold one column and one row
    (1, 17, 21, 10, 33, (3, 3), (0, 0, 0, 0)),       # no padding
    (3, 40, 18, 22, 130, (2, 3), (0, 1, 2, 0)),      # even filter height, left padding of two, none on the right
    (1, 64, 25, 30, 20, (5, 5), (2, 2, 3, 1)),       # 25 taps, odd left padding
    (1, 64, 16, 14, 40, (1, 2), (0, 0, 4, 3)),       # the first pixels see nothing but padding
    (2, 64, 70, 90, 64, (3, 3), (1, 1, 1, 1)),       # several tiles a CTA
]


@pytest.mark.parametrize("orientation", [1, 2])
@pytest.mark.parametrize("geo", GEOMETRIES)
def test_patch_pairs(checker, geo, orientation):
    N, C, H, W, O, k, pad = geo
    tune = dict(patch_mode=2, mma_orientation=orientation)
    shape = (O, C) + k
    plan = ops.ConvPlan((N, C, H, W), shape, pad, (2, 2), (1, 1), **tune)
    assert orientation == 2 or "mode=patch" in plan.describe()      # (a swapped tile of 256 pixels and 128 channels may not fit)
    assert "mode=patch" not in ops.ConvPlan((N, C, H, W + 1), shape, pad, (2, 2), (1, 1), **tune).describe()
    rng = np.random.default_rng(9)
    x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-128, 128, shape).astype(np.int8)
    dq = rng.uniform(1e-4, 1e-3, O).astype(np.float32)
    bias = rng.normal(0, 0.1, O).astype(np.float32)
    rq = [np.float32(2.5)] * N
    y = checker.activation(checker.add_bias(checker.conv2d_quantized(x, w, pad, (2, 2), (1, 1), dq, 0.0), bias), "relu", 0.0)
    for kw in (dict(want_f32=False, rq=rq, i8_layout="nhwc"), dict(), dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc")):
        got = run_gpu(x, w, pad, (2, 2), (1, 1), dq, bias, "relu", 0.0, x_layout="nhwc", want_acc=False, tune=tune, **kw)
        if kw.get("want_f32", True):
            assert same_bits(got["f32"], y)
        if "rq" in kw:
            assert np.array_equal(got["i8"], checker.quantize(y, rq))
