"""The networks' forward() repeats bound library calls: after any change to what a pass is made of they have to be the calls that the
pass as plain code would make.  On the CPU, with plans and library functions that only note the addresses they are given."""
import numpy as np
import pytest
import torch

from tennis_b200 import nets, ops


@pytest.fixture
def noted(monkeypatch):
    log = []

    def note(name):
        def fn(*args):
            log.append((name,) + args)
            return 0
        return fn

    class Plan:
        def __init__(self, *args, **kwargs):
            self.workspace = torch.zeros(64, dtype=torch.uint8)

        def set_weights(self, w, stream=None):
            pass

        def quantize_input(self, x, scales, stream=None):
            log.append(("quantize_input", x.data_ptr(), tuple(scales)))

        def bind(self, *args, **kwargs):
            args = (self,) + args + tuple(kwargs[k] for k in sorted(kwargs))
            at = lambda a: (a.data_ptr() if isinstance(a, torch.Tensor) else a.workspace.data_ptr() if isinstance(a, Plan) else
                            tuple(a) if hasattr(a, "_length_") else a)
            tensors = [a.workspace if isinstance(a, Plan) else a for a in args if isinstance(a, (Plan, torch.Tensor))]
            return ops.Call(note("conv"), tuple(at(a) for a in args), args, tensors)

        bind_run = bind_projected = bind_concat = bind

    class Library:
        def __getattr__(self, name):
            return note(name)

    monkeypatch.setattr(ops, "ConvPlan", Plan)
    monkeypatch.setattr(nets._lib, "load", Library)
    monkeypatch.setattr(ops, "padded_channels", lambda c: c)
    monkeypatch.setattr(ops, "_stream_ptr", lambda stream=None: 0)
    return log


def network(kind):
    if kind == "resnet":
        spec = nets.resnet_spec(image=32, widths=(8, 16), blocks=(2, 1), stem_channels=8, classes=10)
        net = nets.QuantResNet(spec, nets.make_params(spec, 0), 1, device="cpu")
    else:
        spec = nets.cspdarknet_spec(image=32, widths=(8, 16), blocks=(1, 1), stem_channels=8)
        net = nets.QuantCSPDarknet(spec, nets.make_conv_params(spec, 0), 1, device="cpu")
    for i in range(len(net.convs)):
        net._set_in_scale(i, 1.0 + i)
        net._set_out_scale(i, 2.0 + i)
    net.input_scale = 3.0
    net.input_scale_arr = nets._lib.float_array([3.0])
    net.calibrated = True
    return net


def _bias(net):
    net.convs[2]["bias"] = torch.ones(7)


def _bias_data(net):
    net.convs[2]["bias"].data = torch.ones(7)


def _layer(net):
    net.convs[1] = dict(net.convs[1], dq=torch.ones(3))


def _buffer(net):
    key = sorted(net.buffers)[0]
    net.buffers[key] = torch.ones_like(net.buffers[key])


def _buffers(net):
    net.kept, net.buffers = net.buffers, {}


def _buffer_of_new_buffers(net):
    _buffers(net)
    net.forward(torch.zeros(1))
    _buffer(net)


def _workspace(net):
    net.convs[2]["plan"].workspace = torch.zeros(128, dtype=torch.uint8)


CHANGES = dict(in_scale=lambda net: net._set_in_scale(2, 9.0), out_scale=lambda net: net._set_out_scale(2, 9.0), bias=_bias, bias_data=_bias_data,
               layer=_layer, buffer=_buffer, buffers=_buffers, buffer_of_new_buffers=_buffer_of_new_buffers, workspace=_workspace,
               edited=lambda net: net.convs[2].update(dq=torch.ones(7)), fused=lambda net: (setattr(net, "fuse_projection", False), setattr(net, "fuse_concat", False)),
               classifier=lambda net: setattr(net, "fc_w", torch.ones(5)))


@pytest.mark.parametrize("change", sorted(CHANGES))
@pytest.mark.parametrize("kind", ["resnet", "cspdarknet"])
def test_a_changed_network_is_seen_by_the_next_pass(noted, kind, change):
    net = network(kind)
    x = torch.zeros(1)

    def one_pass():
        del noted[:]
        net.forward(x)
        return [c for c in noted]

    first = one_pass()
    assert one_pass() == first and len(first) > 10
    CHANGES[change](net)
    after = one_pass()
    net.steps = None                          # the pass as plain code
    plain = one_pass()
    # (a pass that found an address changed under it has begun once in vain)
    assert after[-len(plain):] == plain and one_pass() == plain


def test_passes_of_unchanged_networks_are_bound(noted):
    net = network("resnet")
    net.forward(torch.zeros(1))
    steps = net.steps
    net.forward(torch.zeros(1))
    assert net.steps is steps


def test_a_network_is_freed_with_its_last_reference(noted):
    import gc
    import weakref
    net = network("resnet")
    net.forward(torch.zeros(1))
    held = weakref.ref(net.buffers["logits"])
    gc.disable()
    try:
        del net
        assert held() is None
    finally:
        gc.enable()
