"""What operator "conv2d_quantized" keeps between calls, on the CPU: the plan is replaced by a convolution in plain torch that
works, as the real one does, from the weights and the geometry it was given."""
import numpy as np
import pytest
import torch

from tennis_b200 import ops


class PlainPlan:
    """Stands in for ops.ConvPlan: the weights are packed (copied) by set_weights, the geometry is fixed when it is made."""

    def __init__(self, xshape, wshape, pad, stride, dilation, padding_value, kernel, device):
        self.pad, self.stride, self.dilation = [tuple(int(v) for v in t) for t in (pad, stride, dilation)]
        kh, kw = [d * (k - 1) + 1 for d, k in zip(self.dilation, wshape[2:])]
        self.out_shape = (xshape[0], wshape[0], (xshape[2] + self.pad[0] + self.pad[1] - kh) // self.stride[0] + 1,
                          (xshape[3] + self.pad[2] + self.pad[3] - kw) // self.stride[1] + 1)

    def set_weights(self, w, stream=None):
        self.packed = w.float().contiguous().clone()

    def run(self, x, x_layout, dq, out_f32=None, out_acc=None, stream=None):
        out_f32.copy_(plain(x, self.packed, dq, self.pad, self.stride, self.dilation))


def plain(x, w, dq, pad, stride, dilation):
    x = torch.nn.functional.pad(x.float(), (pad[2], pad[3], pad[0], pad[1]))
    return torch.nn.functional.conv2d(x, w.float(), None, stride, 0, dilation) * dq.reshape(1, -1, 1, 1)


def operator(monkeypatch, dq, pad=1, stride=1):
    monkeypatch.setattr(ops, "ConvPlan", PlainPlan)
    op = ops.Conv2DQuantized()
    configure(op, dq, pad, stride)
    return op


def configure(op, dq, pad=1, stride=1, fmt="NCHW"):
    op.set("format", fmt)
    spatial = [[0, 0], [0, 0], [pad, pad], [pad, pad]]
    op.set("padding", np.array(spatial if fmt == "NCHW" else spatial[1:] + spatial[:1], dtype=np.int32))
    op.set("stride", np.array([1, 1, stride, stride] if fmt == "NCHW" else [1, stride, stride, 1], dtype=np.int32))
    op.set("dilation", np.array([1, 1, 1, 1], dtype=np.int32))
    op.set("dequantize_scales", np.asarray(dq, dtype=np.float32))
    op.init()


def tensors(seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randint(-8, 8, (2, 4, 7, 6), generator=g, dtype=torch.int8)
    w = torch.randint(-8, 8, (5, 4, 3, 3), generator=g, dtype=torch.int8)
    return x, w, [0.5, 1.0, 2.0, 4.0, 8.0]


def same(got, x, w, dq, pad=1, stride=1):
    return torch.equal(got, plain(x, w, torch.tensor(dq), (pad,) * 4, (stride,) * 2, (1, 1)))


def test_attributes_set_again_take_effect(monkeypatch):
    x, w, dq = tensors()
    op = operator(monkeypatch, dq)
    assert same(op.run([x, w]), x, w, dq)
    dq2 = [2.0, 0.25, 1.0, 1.0, 0.5]
    configure(op, dq2)
    assert same(op.run([x, w]), x, w, dq2)
    configure(op, dq2, pad=0, stride=2)
    assert same(op.run([x, w]), x, w, dq2, pad=0, stride=2)
    configure(op, dq)                         # and back
    assert same(op.run([x, w]), x, w, dq)


def test_attributes_set_again_are_checked_again(monkeypatch):
    x, w, dq = tensors()
    op = operator(monkeypatch, dq)
    op.run([x, w])
    configure(op, dq[:3])
    with pytest.raises(ops.EjectionException):
        op.run([x, w])
    configure(op, dq, fmt="NHWC")
    with pytest.raises(ops.EjectionException):
        op.run([x, w])
    configure(op, dq)
    op.set("padding", np.zeros((3, 2), dtype=np.int32))
    with pytest.raises(ops.EjectionException):
        op.init()


def test_weights_written_between_calls_are_used(monkeypatch):
    x, w, dq = tensors()
    op = operator(monkeypatch, dq)
    op.run([x, w])
    w.neg_()
    assert same(op.run([x, w]), x, w, dq)
    w[:, 1:3].fill_(3)                        # through a view
    assert same(op.run([x, w]), x, w, dq)
    with torch.inference_mode():              # tensors whose writes are not counted
        v = w + 0
        op.run([x, v])
        v.mul_(2)
        assert same(op.run([x, v]), x, v, dq)


def test_views_of_the_same_weights_are_told_apart(monkeypatch):
    x, w, dq = tensors()
    op = operator(monkeypatch, dq)
    assert same(op.run([x, w]), x, w, dq)
    turned = w.transpose(2, 3)
    assert same(op.run([x, turned]), x, turned, dq)
    assert same(op.run([x, w]), x, w, dq)


def test_weights_of_a_plan_stay_allocated(monkeypatch):
    """A later tensor cannot come to lie where the weights of a kept plan were."""
    import weakref
    x, w, dq = tensors()
    op = operator(monkeypatch, dq)
    w = w.transpose(2, 3)
    held = weakref.ref(w)
    op.run([x, w])
    del w
    assert held() is not None


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [1, 2])
def test_attributes_and_weights_on_the_gpu(kernel):
    x, w, dq = tensors()
    x, w = x.cuda(), w.cuda()
    op = ops.Conv2DQuantized(kernel)
    configure(op, dq)
    first = op.run([x, w])
    w.neg_()
    assert torch.equal(op.run([x, w]), -first)
    turned = op.run([x, w.transpose(2, 3)])
    assert torch.equal(turned, op.run([x, w.transpose(2, 3).contiguous()]))
    configure(op, [2 * v for v in dq])
    assert torch.equal(op.run([x, w]), -2 * first)


def test_quantize_takes_scales_as_they_stand():
    op = ops.Quantize()
    op.set("quantize_scale", [1.0, 2.0])
    op.init()
    assert list(op._scale_array()) == [1.0, 2.0]
    op.scales[1] = 4.0
    assert list(op._scale_array()) == [1.0, 4.0]
    op.scales = [3.0]
    assert list(op._scale_array()) == [3.0]
