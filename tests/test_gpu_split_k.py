"""Deep layers of few tiles, whose K blocks four CTAs of a cluster share: exact int32 sums through every epilogue, against the CPU
checker bit for bit.  Shapes at the rule's edges: K of 2048 bytes and just above, block counts that four does not divide, channel tiles that
end inside a 32-channel chunk, the last pixel tile nearly empty, 64-byte K blocks, the most tiles that are still split."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from test_gpu_conv import run_gpu
from tennis_b200 import ops

pytestmark = pytest.mark.gpu

# N, C, H, W, O, K, stride, pad
GEOMETRIES = [
    (1, 2048, 7, 7, 64, 1, 1, 0),        # 16 K blocks, one tile, half of its channels
    (2, 2049, 5, 13, 130, 1, 1, 0),      # 33 blocks of 64, two channel tiles, the second with two channels
    (1, 512, 9, 15, 85, 3, 1, 1),        # 135 pixels: the second pixel tile holds seven; ragged chunk
    (3, 576, 11, 10, 100, 3, 2, 1),      # 81 blocks of 64, strided; O % 4 == 0
    (1, 200, 8, 8, 33, 5, 1, 2),         # 50 blocks, one full chunk and one channel
    (2, 512, 32, 32, 256, 3, 1, 1),      # 16 x 2 tiles: 128 CTAs
]


@pytest.mark.parametrize("outputs", ["i8", "f32", "nhwc", "nhwc_residual", "acc"])
@pytest.mark.parametrize("geo", GEOMETRIES)
def test_split_k(checker, geo, outputs):
    N, C, H, W, O, K, stride, pad = geo
    plan = ops.ConvPlan((N, C, H, W), (O, C, K, K), (pad,) * 4, (stride,) * 2, (1, 1))
    assert "mode=split" in plan.describe()
    rng = np.random.default_rng(7)
    x = rng.integers(-128, 128, (N, C, H, W)).astype(np.int8)
    w = rng.integers(-128, 128, (O, C, K, K)).astype(np.int8)
    dq = rng.uniform(1e-4, 1e-3, O).astype(np.float32)
    bias = rng.normal(0, 0.1, O).astype(np.float32)
    rq = [np.float32(1.3)] * N
    acc = checker.conv2d_quantized(x, w, (pad,) * 4, (stride,) * 2, (1, 1), dq, 0.0)
    y = checker.add_bias(acc, bias)
    res = None
    if outputs == "nhwc_residual":
        res = rng.normal(0, 1, y.shape).astype(np.float32)
        y = y + res
    y = checker.activation(y, "relu", 0.0)
    kw = dict(i8=dict(want_f32=False, rq=rq, i8_layout="nhwc"), f32=dict(), nhwc=dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc"),
              nhwc_residual=dict(rq=rq, i8_layout="nhwc", f32_layout="nhwc", residual=res), acc=dict(want_acc=True, rq=rq))[outputs]
    kw.setdefault("want_acc", False)
    got = run_gpu(x, w, (pad,) * 4, (stride,) * 2, (1, 1), dq, bias, "relu", 0.0, x_layout="nhwc", **kw)
    if outputs == "acc":      # (whole numbers: exact in fp64 in any order)
        sums = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(w).double(), stride=stride, padding=pad)
        assert np.array_equal(got["acc"], sums.numpy().astype(np.int32))
    if kw.get("want_f32", True):
        assert same_bits(got["f32"], y)
    if "rq" in kw:
        assert np.array_equal(got["i8"], checker.quantize(y, rq))
