"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more from the same ranges,
``prepare(case, seed)`` what a program holds before the call (inputs, weights, plans), ``run(state)`` one pass through the
public entry points, ``work(case)`` the bytes and operations the pass cannot do without, ``tolerance(case)`` how far the
outputs of a correct implementation may lie from each other.

Kinds of case:

* ``layer``      one quantized convolution on its plan: fp32 NCHW in, quantize, convolution, bias, activation, fp32 NCHW out;
* ``inner``      the same layer inside a network: int8 NHWC_PAD in, requantized int8 NHWC_PAD out;
* ``operators``  the layer as a module runs it operator by operator: quantize, conv2d_quantized, add_bias, activation;
* ``sweep``      the five layers of the shape sweep, one after the other;
* ``quantize``   the operator ``quantize`` alone (one scale per sample);
* ``host``       the layer on tensors in pinned host memory, through the waiting host-buffer call;
* ``resnet50``, ``cspdarknet53``   a forward pass of the network, as plain calls or as a replayed CUDA graph.
"""
import ctypes
import math

import numpy as np
import torch

from tennis_b200 import _lib, nets, ops, workloads

# value distributions of the benchmark configurations: activations N(0,1) or U(0,1), weights uniform in [-127,127],
# per-channel weight scales U(0.001,0.01), bias N(0,0.1)
_ACT = {"none": _lib.ACT_NONE, "relu": _lib.ACT_RELU, "leaky": _lib.ACT_LEAKY_RELU}
_LEAKY = 0.1
# no drawn case is dearer than the dearest listed one (the CSPDarknet backbone on 16 images)
_MOST_VALUES = 32 << 20          # values of one fp32 tensor
_MOST_OPS = 4e11


def _layer(name, kind, n, c, h, w, o, k, stride=1, dilation=1, act="relu"):
    return dict(name=name, kind=kind, n=n, c=c, h=h, w=w, o=o, k=k, stride=stride, dilation=dilation, act=act)


def listed():
    return [
        # one layer on one image, what an interactive caller waits for: two launches, all latency
        _layer("layer_3x3_64_56_b1", "layer", 1, 64, 56, 56, 64, 3),
        # a layer with channel counts and an image that fit no tile, as exported detection models have them
        _layer("layer_ragged_75_85_b5", "layer", 5, 75, 37, 53, 85, 3, act="leaky"),
        # a wide 1x1 layer inside a network (a plain int8 matrix product): as much arithmetic as one layer has in earnest
        _layer("inner_1x1_2048_32_b8", "inner", 8, 2048, 32, 32, 2048, 1),
        # a module that was not rewritten: the operators run one by one, fp32 and int8 NCHW tensors between them
        _layer("operators_3x3_128_28_b32", "operators", 32, 128, 28, 28, 128, 3),
        # the layer shapes of the benchmark's sweep at its batch: 1x1, 3x3, strided 3x3, deep 1x1, 7x7 stem
        dict(name="sweep_b32", kind="sweep", n=32),
        # quantize alone on a large tensor: pure memory traffic
        dict(name="quantize_64Mi", kind="quantize", n=64, per_sample=1 << 20, dtype="float32"),
        # the layer called with CPU-resident tensors: upload, two kernels, download, wait
        _layer("host_3x3_128_28_b32", "host", 32, 128, 28, 28, 128, 3),
        # a classification network: one image at a time by plain calls, a small batch and the benchmark's batch as graphs
        dict(name="resnet50_b1_calls", kind="resnet50", n=1, image=224, graph=False),
        dict(name="resnet50_b8_graph", kind="resnet50", n=8, image=224, graph=True),
        dict(name="resnet50_b64_graph", kind="resnet50", n=64, image=224, graph=True),
        # a detection backbone: one image, and the benchmark's batch of large images
        dict(name="cspdarknet53_b1_graph", kind="cspdarknet53", n=1, image=608, graph=True),
        dict(name="cspdarknet53_b16_calls", kind="cspdarknet53", n=16, image=608, graph=False),
    ]


def _log(rng, lo, hi):
    """An integer from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """A channel count: mostly a multiple of 16 as networks have them, sometimes any number."""
    c = _log(rng, lo, hi)
    return c if rng.random() < 0.35 or c < 16 else max(lo, c // 16 * 16)


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "inner", "inner", "operators", "quantize", "host", "resnet50", "cspdarknet53"])
    if kind == "quantize":
        n = _log(rng, 1, 128)
        return dict(kind=kind, n=n, per_sample=max(1, _log(rng, 1 << 12, 64 << 20) // n), dtype=rng.choice(["float32", "float32", "float32", "float64"]))
    if kind == "resnet50":
        return dict(kind=kind, n=_log(rng, 1, 64), image=32 * rng.randint(4, 8), graph=rng.random() < 0.6)
    if kind == "cspdarknet53":
        image = 32 * rng.randint(8, 19)
        return dict(kind=kind, n=_log(rng, 1, 8), image=image, graph=rng.random() < 0.6)
    while True:
        k = rng.choice([1, 1, 3, 3, 3, 5, 7])
        case = dict(kind=kind, n=_log(rng, 1, 64), c=_channels(rng, 17 if kind == "inner" else 3, 2048), h=_log(rng, 7, 224), w=0,
                    o=_channels(rng, 8, 2048), k=k, stride=rng.choice([1, 1, 2]), dilation=2 if k == 3 and rng.random() < 0.15 else 1,
                    act=rng.choice(["relu", "relu", "leaky", "none"]))
        case["w"] = case["h"] if rng.random() < 0.6 else _log(rng, 7, 224)
        geo = _geometry(case)
        values = max(case["n"] * case["c"] * case["h"] * case["w"], case["n"] * case["o"] * geo["oh"] * geo["ow"])
        if kind == "host":
            values *= 16             # these bytes cross the host link
        if values <= _MOST_VALUES and geo["ops"] <= _MOST_OPS and case["o"] * case["c"] * k * k <= 16 << 20:
            return case


def _geometry(case):
    pad = case["dilation"] * (case["k"] - 1) // 2
    oh = ops.conv_out_dim(case["h"], pad, pad, case["k"], case["stride"], case["dilation"])
    ow = ops.conv_out_dim(case["w"], pad, pad, case["k"], case["stride"], case["dilation"])
    return dict(pad=pad, oh=oh, ow=ow, ops=2.0 * case["n"] * case["o"] * oh * ow * case["c"] * case["k"] * case["k"])


def _sweep_cases(n):
    return [dict(kind="layer", n=n, c=l["c"], h=l["h"], w=l["w"], o=l["o"], k=l["kh"], stride=l["stride"], dilation=l["dilation"], act=l["act"])
            for l in workloads.CONFIG1]


# ---- what a program holds before the call ---------------------------------------------------------------------------
def _layer_state(case, gen):
    dev = torch.device("cuda")
    n, c, h, w, o, k = (case[v] for v in ("n", "c", "h", "w", "o", "k"))
    pad = _geometry(case)["pad"]
    x = torch.randn((n, c, h, w), device=dev, generator=gen)
    qscale = np.float32(127.0) / np.float32(float(x.abs().max()))
    wgt = torch.randint(-127, 128, (o, c, k, k), device=dev, generator=gen, dtype=torch.int8)
    sw = torch.empty(o, device=dev).uniform_(0.001, 0.01, generator=gen)
    bias = torch.empty(o, device=dev).normal_(0.0, 0.1, generator=gen)
    st = dict(kind=case["kind"], act=_ACT[case["act"]], x=x, w=wgt, bias=bias, dq=sw / float(qscale), qscale=float(qscale), n=n, pad=pad,
              stride=case["stride"], dilation=case["dilation"])
    return st


def _make_plan(st):
    return ops.ConvPlan(tuple(st["x"].shape), tuple(st["w"].shape), (st["pad"],) * 4, (st["stride"],) * 2, (st["dilation"],) * 2)


def _prepare_layer(case, gen):
    st = _layer_state(case, gen)
    st["plan"] = _make_plan(st)
    st["plan"].set_weights(st["w"])
    st["scales"] = _lib.float_array([st["qscale"]] * st["n"])
    st["out"] = torch.empty(st["plan"].out_shape, dtype=torch.float32, device="cuda")
    return st


def _prepare_inner(case, gen):
    st = _layer_state(case, gen)
    plan = st["plan"] = _make_plan(st)
    plan.set_weights(st["w"])
    st["xq"] = ops.quantize_nchw_to_nhwc(st["x"], [st["qscale"]] * st["n"])
    # the requantize scale a calibration would have chosen: 127 / max of the layer's fp32 output
    f = torch.empty(plan.out_shape, dtype=torch.float32, device="cuda")
    plan.run(st["xq"], _lib.LAYOUT_NHWC_PAD, st["dq"], bias=st["bias"], activation=st["act"], leaky=_LEAKY, out_f32=f)
    top = float(f.abs().max())
    st["requant"] = _lib.float_array([127.0 / top if top > 0 else 1.0] * st["n"])
    n, o, oh, ow = plan.out_shape
    st["out"] = torch.empty((n, oh, ow, ops.padded_channels(o)), dtype=torch.int8, device="cuda")
    del st["x"]
    return st


def _prepare_operators(case, gen):
    st = _layer_state(case, gen)
    st["quantize"] = q = ops.Quantize()
    q.set("quantize_scale", np.full(st["n"], st["qscale"], dtype=np.float32))
    q.init()
    st["conv"] = op = ops.Conv2DQuantized()
    p, s, d = st["pad"], st["stride"], st["dilation"]
    op.set("format", "NCHW")
    op.set("padding", np.array([[0, 0], [0, 0], [p, p], [p, p]], dtype=np.int32))
    op.set("stride", np.array([1, 1, s, s], dtype=np.int32))
    op.set("dilation", np.array([1, 1, d, d], dtype=np.int32))
    op.set("dequantize_scales", st["dq"].cpu().numpy())
    op.init()
    return st


def _prepare_host(case, gen):
    st = _layer_state(case, gen)
    plan = st["plan"] = _make_plan(st)
    for name in ("x", "w", "dq", "bias"):
        st[name] = st[name].cpu().pin_memory()
    st["scales"] = _lib.float_array([st["qscale"]] * st["n"])
    st["out"] = torch.zeros(plan.out_shape, dtype=torch.float32).pin_memory()
    size = _lib.load().tsb_conv2d_host_scratch_bytes(plan.handle)
    st["scratch"] = torch.empty(size, dtype=torch.uint8, device="cuda")
    st["args"] = (plan.handle, st["x"].data_ptr(), st["scales"], st["n"], st["w"].data_ptr(), ctypes.cast(st["dq"].data_ptr(), ctypes.c_void_p),
                  st["bias"].data_ptr(), st["act"], _LEAKY, st["out"].data_ptr(), st["scratch"].data_ptr(), size)
    _call_host(st, 0)                      # the weights go up once and stay
    return st


def _prepare_net(case, gen, seed):
    n, image = case["n"], case["image"]
    fuse = n > 1          # the two-in-one launches take one scale per image of a batch, not the single-scale rounding of one image
    if case["kind"] == "resnet50":
        spec = nets.resnet_spec(image=image)
        net = nets.QuantResNet(spec, nets.make_params(spec, seed), n, fuse_projection=fuse)
        x = torch.randn((n, 3, image, image), device="cuda", generator=gen)
    else:
        spec = nets.cspdarknet_spec(image=image)
        net = nets.QuantCSPDarknet(spec, nets.make_conv_params(spec, seed), n, fuse_concat=fuse)
        x = torch.rand((n, 3, image, image), device="cuda", generator=gen)
    net.calibrate(x)
    st = dict(kind=case["kind"], net=net, x=x, graph=None)
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            net.forward(x)
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            st["out"] = net.forward(x)
    return st


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "layer":
        return _prepare_layer(case, gen)
    if kind == "inner":
        return _prepare_inner(case, gen)
    if kind == "operators":
        return _prepare_operators(case, gen)
    if kind == "host":
        return _prepare_host(case, gen)
    if kind == "sweep":
        return dict(kind=kind, layers=[_prepare_layer(c, gen) for c in _sweep_cases(case["n"])])
    if kind == "quantize":
        x = torch.randn((case["n"], case["per_sample"]), device="cuda", generator=gen, dtype=getattr(torch, case["dtype"]))
        op = ops.Quantize()
        op.set("quantize_scale", (127.0 / x.abs().amax(dim=1).clamp_min(1e-6)).float().cpu().numpy())
        op.init()
        return dict(kind=kind, op=op, x=x)
    return _prepare_net(case, gen, int(seed))


# ---- one pass -------------------------------------------------------------------------------------------------------
def _run_layer(st):
    plan = st["plan"]
    plan.quantize_input(st["x"], st["scales"])
    plan.run(None, _lib.LAYOUT_STAGED, st["dq"], bias=st["bias"], activation=st["act"], leaky=_LEAKY, out_f32=st["out"])
    return st["out"]


def _call_host(st, resident):
    _lib.check(_lib.load().tsb_conv2d_quantized_host(*st["args"], resident, torch.cuda.current_stream().cuda_stream))


def run(state):
    kind = state["kind"]
    if kind == "layer":
        return _run_layer(state)
    if kind == "inner":
        state["plan"].run(state["xq"], _lib.LAYOUT_NHWC_PAD, state["dq"], bias=state["bias"], activation=state["act"], leaky=_LEAKY,
                          out_i8=state["out"], out_i8_layout=_lib.LAYOUT_NHWC_PAD, requant_scales=state["requant"])
        return state["out"]
    if kind == "operators":
        q = state["quantize"].run([state["x"]])
        y = ops.add_bias(state["conv"].run([q, state["w"]]), state["bias"])
        if state["act"] == _lib.ACT_RELU:
            y = ops.relu(y)
        elif state["act"] == _lib.ACT_LEAKY_RELU:
            y = ops.leaky_relu(y, _LEAKY)
        return [q, y]
    if kind == "sweep":
        return [_run_layer(st) for st in state["layers"]]
    if kind == "quantize":
        return state["op"].run([state["x"]])
    if kind == "host":
        _call_host(state, 1)
        return state["out"]
    if state["graph"] is not None:
        state["graph"].replay()
        return state["out"]
    return state["net"].forward(state["x"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _layer_work(case):
    geo = _geometry(case)
    n, c, o = case["n"], case["c"], case["o"]
    pixels_in, pixels_out = n * case["h"] * case["w"], n * geo["oh"] * geo["ow"]
    weights = o * c * case["k"] * case["k"] + 8 * o
    if case["kind"] == "inner":
        return dict(bytes=pixels_in * c + weights + pixels_out * o, flops=geo["ops"])
    more = pixels_in * c if case["kind"] == "operators" else 0        # the int8 tensor is an output too
    return dict(bytes=4 * pixels_in * c + more + weights + 4 * pixels_out * o, flops=geo["ops"])


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        parts = [_layer_work(c) for c in _sweep_cases(case["n"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "quantize":
        return dict(bytes=(5 if case["dtype"] == "float32" else 9) * case["n"] * case["per_sample"], flops=2 * case["n"] * case["per_sample"])
    if kind not in ("resnet50", "cspdarknet53"):
        return _layer_work(case)
    n, image = case["n"], case["image"]
    if kind == "resnet50":
        spec = nets.resnet_spec(image=image)
        head = spec["classes"] * spec["features"]
        extra, flops = 4 * head + 4 * spec["classes"] * (n + 1), 2.0 * n * head
    else:
        spec = nets.cspdarknet_spec(image=image)
        extra, flops = n * spec["final_size"] ** 2 * spec["features"], 0.0
    weights = sum(c["o"] * c["c"] * c["k"] * c["k"] + 8 * c["o"] for c in spec["convs"])
    return dict(bytes=12 * n * image * image + weights + extra, flops=flops + nets.conv_ops(spec, n))


def tolerance(case):
    # int8 outputs are whole numbers; the fp32 output of a layer is an exact int32 sum followed by separately rounded fp32
    # steps in a fixed order, so its bits are given as well.  The network's logits are fp32 sums over 49 pixels and 2048
    # features, free in their order.
    return {"rel": 1e-5} if case["kind"] == "resnet50" else "exact"
