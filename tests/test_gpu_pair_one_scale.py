"""The two-in-one launches (projected shortcut, concatenated input) requantized with ONE scale: half to even, half away from zero in the
tensor's last count % 8 elements.  Bit for bit against the CPU checker's operator chain; scales and biases are powers of two, so that exact
ties are frequent.  And networks of one image, which take these launches by default, against the whole chain."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from test_gpu_projected import expected, run_projected
import test_gpu_csp
import test_gpu_resnet

pytestmark = pytest.mark.gpu


def tie_data(rng, O):
    return np.float32(2.0) ** rng.integers(-6, -3, O).astype(np.float32), (rng.integers(-8, 9, O) / 4).astype(np.float32)


# N, C (main), C (shortcut), H, W (output grid), O, shortcut stride, tile_channels
PROJECTED = [
    (1, 64, 64, 12, 12, 64, 1, 0),         # no tail
    (1, 64, 128, 7, 9, 100, 2, 0),         # tail of four, last chunk of four channels
    (1, 128, 64, 7, 7, 260, 1, 256),       # two channel tiles, the second of four channels
    (3, 64, 64, 5, 5, 100, 1, 128),        # several images under one scale
    (41, 64, 64, 13, 13, 260, 1, 128),     # several tiles per CTA, a tail in the last
]


@pytest.mark.parametrize("variant", ["both", "i8", "after"])
@pytest.mark.parametrize("case", PROJECTED)
def test_projected_shortcut(checker, case, variant):
    N, C, Cs, H, W, O, stride, tile = case
    rng = np.random.default_rng(sum(case))
    x = rng.integers(-20, 21, (N, C, H, W), dtype=np.int8)
    xs = rng.integers(-20, 21, (N, Cs, (H - 1) * stride + 1, (W - 1) * stride + 1), dtype=np.int8)
    w, ws = rng.integers(-3, 4, (O, C, 1, 1), dtype=np.int8), rng.integers(-3, 4, (O, Cs, 1, 1), dtype=np.int8)
    (dq, bias), (dqs, bias_s) = tie_data(rng, O), tie_data(rng, O)
    act, leaky, after = ("leaky_relu", 0.25, True) if variant == "after" else ("relu", 0.0, False)
    rq = [np.float32(1.0)]
    want_f, want_q = expected(checker, x, w, xs, ws, (stride, stride), dq, bias, dqs, bias_s, act, leaky, rq, after)
    got = run_projected(x, w, xs, ws, (stride, stride), dq, bias, dqs, bias_s, act, leaky, rq, res_after=after, tile_channels=tile,
                        want_f32=variant != "i8")
    if variant != "i8":
        assert same_bits(got["f32"], want_f)
    assert np.array_equal(got["i8"], want_q)


# N, C_first, C_rest, H, W, O, tile_channels
CONCAT = [
    (1, 64, 64, 12, 12, 64, 0),
    (1, 128, 64, 7, 9, 100, 0),
    (1, 64, 128, 7, 7, 260, 256),
    (3, 64, 64, 5, 5, 20, 0),              # a narrow tile, one chunk of twenty channels
    (41, 64, 64, 13, 13, 260, 0),
]


@pytest.mark.parametrize("far", [False, True])           # far: values beyond the int32 range, which go element by element
@pytest.mark.parametrize("outputs", ["i8", "both"])
@pytest.mark.parametrize("case", CONCAT)
def test_concatenated_input(checker, case, outputs, far):
    from tennis_b200 import ops
    N, C1, C2, H, W, O, tile = case
    rng = np.random.default_rng(sum(case))
    x1, x2 = rng.integers(-20, 21, (N, C1, H, W), dtype=np.int8), rng.integers(-20, 21, (N, C2, H, W), dtype=np.int8)
    w = rng.integers(-3, 4, (O, C1 + C2, 1, 1), dtype=np.int8)
    dq, bias = tie_data(rng, O)
    if far:
        bias[::7] = 3e9
    rq = [np.float32(1.0)]
    y = checker.conv2d_quantized(np.concatenate([x1, x2], axis=1), w, (0,) * 4, (1, 1), (1, 1), dq, 0.0)
    y = checker.activation(checker.add_bias(y, bias), "leaky_relu", 0.25)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    first, rest = [ops.ConvPlan(v.shape, (O, v.shape[1], 1, 1), (0,) * 4, (1, 1), (1, 1), 0.0, 2, "cuda") for v in (x1, x2)]
    first.set_weights(t(w[:, :C1]))
    rest.set_weights(t(w[:, C1:]))
    out_f32 = torch.full((N, H, W, O), float("nan"), dtype=torch.float32, device="cuda") if outputs == "both" else None
    out_i8 = torch.full((N, H, W, ops.padded_channels(O)), 99, dtype=torch.int8, device="cuda")
    rest.run_concat(ops.repack_nchw_to_nhwc(t(x2)), first, ops.repack_nchw_to_nhwc(t(x1)), t(dq), bias=t(bias), activation=2, leaky=0.25,
                    out_f32=out_f32, out_i8=out_i8, requant_scales=rq, tile_channels=tile)
    rest.status()
    if out_f32 is not None:
        assert same_bits(out_f32.cpu().numpy().transpose(0, 3, 1, 2), y)
    q = out_i8.cpu().numpy()
    assert not q[..., O:].any()
    assert np.array_equal(q[..., :O].transpose(0, 3, 1, 2), checker.quantize(y, rq))


def test_values_beyond_int32_through_a_projection(checker):
    rng = np.random.default_rng(5)
    x, xs = rng.integers(-20, 21, (1, 64, 5, 5), dtype=np.int8), rng.integers(-20, 21, (1, 64, 5, 5), dtype=np.int8)
    w, ws = rng.integers(-3, 4, (100, 64, 1, 1), dtype=np.int8), rng.integers(-3, 4, (100, 64, 1, 1), dtype=np.int8)
    (dq, bias), (dqs, bias_s) = tie_data(rng, 100), tie_data(rng, 100)
    bias_s[::7] = 3e9
    rq = [np.float32(1.0)]
    want_f, want_q = expected(checker, x, w, xs, ws, (1, 1), dq, bias, dqs, bias_s, "none", 0.0, rq, False)
    got = run_projected(x, w, xs, ws, (1, 1), dq, bias, dqs, bias_s, "none", 0.0, rq)
    assert same_bits(got["f32"], want_f) and np.array_equal(got["i8"], want_q)


@pytest.mark.parametrize("fused", [True, False])
def test_networks_of_one_image(checker, fused):
    from tennis_b200 import nets
    rng = np.random.default_rng(2)
    spec = nets.resnet_spec(image=64, widths=(64, 128), blocks=(2, 1), classes=10)
    params = nets.make_params(spec, seed=1)
    x = rng.standard_normal((1, 3, 64, 64), dtype=np.float32)
    xd = torch.from_numpy(x).cuda()
    net = nets.QuantResNet(spec, params, 1, fuse_projection=fused)
    scales = net.calibrate(xd)
    logits = net.forward(xd).clone()
    assert torch.equal(net.forward(xd), logits)              # (the bound calls)
    net.status()
    outs, last_f32, want = test_gpu_resnet.reference_forward(spec, params, scales, x, checker)
    blocks = [b for stage in spec["stages"] for b in stage]
    for b, y in zip(blocks, outs):
        got = net.buffers[b["name"] + ".y.i8"].cpu().numpy()
        assert np.array_equal(got[..., :y.shape[1]].transpose(0, 3, 1, 2), y), b["name"]
    assert same_bits(net.buffers[blocks[-1]["name"] + ".y.f32"].cpu().numpy().transpose(0, 3, 1, 2), last_f32)
    # (fp32 sums over pixels and features in another order)
    np.testing.assert_allclose(logits.cpu().numpy(), want, rtol=1e-5, atol=1e-5 * np.abs(want).max())

    spec = nets.cspdarknet_spec(image=64, widths=(64, 128), blocks=(1, 2))
    params = nets.make_conv_params(spec, seed=4)
    x = rng.random((1, 3, 64, 64), dtype=np.float32)
    xd = torch.from_numpy(x).cuda()
    net = nets.QuantCSPDarknet(spec, params, 1, fuse_concat=fused)
    scales = net.calibrate(xd)
    out = net.forward(xd).clone()
    assert torch.equal(net.forward(xd), out)
    net.status()
    _, last = test_gpu_csp.reference_forward(spec, params, scales, x, checker)
    assert np.array_equal(out.cpu().numpy()[..., :spec["features"]].transpose(0, 3, 1, 2), last)
