"""Requantize with one scale (a batch of one: half to even, but half away from zero in the tensor's last count % 8 elements) and
channel / pixel counts that end inside a 32-column chunk, through every epilogue of a plain convolution, against the CPU
checker: bit for bit.  Scales and biases are powers of two, so that about one value in eight is an exact tie."""
import numpy as np
import pytest

from conftest import same_bits
from test_gpu_conv import run_gpu

pytestmark = pytest.mark.gpu

# N, C, H, W, O, K, stride, pad, tune
GEOMETRIES = [
    (1, 64, 12, 12, 64, 1, 1, 0, {}),                              # plain tiles; count a multiple of 8: no tail
    (1, 64, 13, 11, 85, 1, 1, 0, {}),                              # tail of 3, last chunk of 21 channels
    (1, 64, 9, 9, 260, 1, 1, 0, {}),                               # tail of 4, O % 4 == 0: staged tiles, two channel tiles
    (3, 128, 7, 7, 129, 3, 1, 1, {}),                              # several images under one scale, tail of 3
    (1, 64, 19, 17, 33, 3, 1, 1, dict(patch_mode=2)),              # patch mode, ragged tiles
    (1, 64, 19, 17, 33, 3, 1, 1, dict(mma_orientation=2)),         # channels on the MMA's M side
    (1, 64, 19, 17, 33, 3, 1, 1, dict(mma_orientation=2, patch_mode=2)),
    (2, 64, 11, 13, 20, 3, 2, 1, dict(mma_orientation=2)),         # 42 pixels an image: chunks cross images and end early
    (1, 3, 20, 132, 13, 3, 1, 1, dict(raw_row_mode=2)),            # raw rows, 16 padded channels
    (1, 64, 1, 1, 5, 1, 1, 0, {}),                                 # five values: nothing but tail
]


def data(geo, seed, n_scales):
    N, C, H, W, O, K, stride, pad, tune = geo
    rng = np.random.default_rng(seed)
    x = rng.integers(-20, 21, (N, C, H, W), dtype=np.int8)
    w = rng.integers(-3, 4, (O, C, K, K), dtype=np.int8)
    dq = np.float32(2.0) ** rng.integers(-4, -1, O).astype(np.float32)
    bias = (rng.integers(-8, 9, O) / 4).astype(np.float32)
    return x, w, (pad,) * 4, (stride,) * 2, dq, bias, [np.float32(1.0)] * n_scales


@pytest.mark.parametrize("act", ["none", "relu", "leaky_relu"])
@pytest.mark.parametrize("outputs", ["i8", "f32", "nhwc", "nhwc_residual"])
@pytest.mark.parametrize("geo", GEOMETRIES)
def test_one_scale(checker, geo, outputs, act):
    x, w, pad, stride, dq, bias, rq = data(geo, 11, 1)
    leaky = 0.25 if act == "leaky_relu" else 0.0
    y = checker.add_bias(checker.conv2d_quantized(x, w, pad, stride, (1, 1), dq, 0.0), bias)
    res, after = None, act == "leaky_relu"
    if outputs == "nhwc_residual":
        res = (np.random.default_rng(12).integers(-40, 41, y.shape) / 8).astype(np.float32)
    if res is not None and not after:
        y = y + res
    y = checker.activation(y, act, leaky)
    if res is not None and after:
        y = y + res
    kw = dict(i8=dict(want_f32=False, rq=rq, i8_layout="nhwc"), f32=dict(), nhwc=dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc"),
              nhwc_residual=dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc", residual=res, res_after=after))[outputs]
    got = run_gpu(x, w, pad, stride, (1, 1), dq, bias, act, leaky, x_layout="nhwc" if x.shape[1] > 16 else "nchw", want_acc=False, tune=geo[-1], **kw)
    if kw.get("want_f32", True):
        assert same_bits(got["f32"], y)
    if "rq" in kw:
        assert np.array_equal(got["i8"], checker.quantize(y, rq))
