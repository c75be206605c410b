"""Pixel-major fp32 tensors of raw-row layers whose weights and image rows leave no shared memory for the staged epilogue: bit for bit
against the CPU checker, one scale (with its tail) or one per image, and no slower than a few times the NCHW output."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from test_gpu_conv import run_gpu
from tennis_b200 import ops

pytestmark = pytest.mark.gpu

# N, C, H, W, O, K, stride, dilation
GEOMETRIES = [
    (1, 3, 35, 416, 96, 5, 1, 1),      # every chunk full
    (1, 3, 29, 509, 100, 5, 1, 1),     # last chunk of four channels, count % 8 != 0: a tail
    (2, 4, 18, 412, 164, 3, 1, 2),     # 256-channel tile
    (2, 3, 42, 704, 164, 7, 2, 1),     # two 8-byte pixels a step
    (1, 3, 51, 608, 12, 9, 2, 1),      # one chunk, twelve channels
]


def plan_of(geo):
    N, C, H, W, O, K, stride, dil = geo
    return ops.ConvPlan((N, C, H, W), (O, C, K, K), (dil * (K // 2),) * 4, (stride,) * 2, (dil,) * 2, device="cpu")


@pytest.mark.parametrize("act", ["relu", "leaky_relu", "none"])
@pytest.mark.parametrize("outputs", ["f32", "both", "residual", "residual_i8", "one_scale"])
@pytest.mark.parametrize("geo", GEOMETRIES)
def test_rows_without_room_for_the_staged_epilogue(checker, geo, outputs, act):
    text = plan_of(geo).describe()
    assert "mode=rows" in text and "staged" not in text
    N, C, H, W, O, K, stride, dil = geo
    pad, after, leaky = (dil * (K // 2),) * 4, act == "leaky_relu", 0.25 if act == "leaky_relu" else 0.0
    rng = np.random.default_rng(3)
    x = rng.integers(-20, 21, (N, C, H, W), dtype=np.int8)
    w = rng.integers(-3, 4, (O, C, K, K), dtype=np.int8)
    dq = np.float32(2.0) ** rng.integers(-6, -3, O).astype(np.float32)      # (ties of the requantize are then exact and frequent)
    bias = (rng.integers(-8, 9, O) / 4).astype(np.float32)
    y = checker.add_bias(checker.conv2d_quantized(x, w, pad, (stride,) * 2, (dil,) * 2, dq, 0.0), bias)
    res = (rng.integers(-40, 41, y.shape) / 8).astype(np.float32) if outputs.startswith("residual") else None
    if res is not None and not after:
        y = y + res
    y = checker.activation(y, act, leaky)
    if res is not None and after:
        y = y + res
    rq = None if outputs == "f32" else [np.float32(1.0)] * (1 if outputs == "one_scale" else N)
    kw = dict(rq=rq, i8_layout="nhwc") if rq else {}
    got = run_gpu(x, w, pad, (stride,) * 2, (dil,) * 2, dq, bias, act, leaky, want_acc=False, f32_layout="nhwc", residual=res, res_after=after,
                  want_f32=outputs != "residual_i8", **kw)
    if outputs != "residual_i8":
        assert same_bits(got["f32"], y)
    if rq:
        assert np.array_equal(got["i8"], checker.quantize(y, rq))


def test_pixel_major_output_costs_about_what_nchw_does():
    N, C, H, W, O, K = 4, 3, 200, 416, 96, 5
    plan = ops.ConvPlan((N, C, H, W), (O, C, K, K), (2,) * 4, (1, 1), (1, 1))
    assert "mode=rows" in plan.describe() and "staged" not in plan.describe()
    plan.set_weights(torch.randint(-100, 100, (O, C, K, K), dtype=torch.int8, device="cuda"))
    plan.quantize_input(torch.randn((N, C, H, W), device="cuda"), [30.0] * N)
    dq = torch.full((O,), 1e-3, device="cuda")
    out = torch.empty(plan.out_shape, device="cuda")

    def shortest(layout):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.run(None, 2, dq, out_f32=out, out_f32_layout=layout)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    nchw, nhwc = shortest(0), shortest(1)
    print("NCHW %.1f us, pixel-major %.1f us" % (nchw * 1e3, nhwc * 1e3))
    assert nhwc < 4 * nchw        # 78 and 38 us; element by element it was 312
