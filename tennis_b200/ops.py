"""Python mirror of the two TenniS operators on the path, over the C ABI.

The shipping host side is the C++ plugin in tennis_b200/plugin/ (TS_REGISTER_OPERATOR on device "gpu"); this
module states the same interface for Python callers and for the parity tests: same operator names, same
attribute names and meaning, the same checks in ``init`` / ``infer`` and the same error texts as

* ts::base::Quantize          src/backend/base/base_quantize.cpp:12-49
* ts::base::Conv2DQuantized   src/backend/base/base_conv2d_quantized.cpp:13-219
* ts::Operator                src/runtime/operator.cpp:22-128 (fields, set, check_params)

Tensors are torch CUDA tensors used as device buffers; all arithmetic happens in libtennis_b200.so.
"""
import ctypes
import operator

import numpy as np
import torch

from . import _lib
from ._lib import (ACT_LEAKY_RELU, ACT_NONE, ACT_RELU, KERNEL_AUTO, KERNEL_DIRECT, KERNEL_TCGEN05, LAYOUT_NCHW,
                   LAYOUT_NHWC_PAD, LAYOUT_STAGED, ConvDesc, ConvEpilogue, TsbError, check, float_array)

REQUIRED, OPTIONAL = "required", "optional"


class EjectionException(RuntimeError):
    """What TS_LOG_ERROR << ... << eject raises in the reference (include/utils/log.h:162-166)."""


# The raw handle of the current stream.  A small convolution takes the GPU 4 us and the driver 3 us to launch;
# torch.cuda.current_stream() builds a Stream object for 3 us more, these two calls take 0.2 us.
_current_device = getattr(torch._C, "_cuda_getDevice", None)
_current_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr(stream=None):
    if stream is None:
        return _current_raw_stream(_current_device())
    return stream.cuda_stream


def _ptr(t):
    return t.data_ptr() if t is not None else None


def padded_channels(c):
    return _lib.load().tsb_padded_channels(int(c))


def conv_out_dim(x, pad_lo, pad_hi, k, stride, dilation):
    """include/backend/common_function.h:30-40: integer division truncating toward zero."""
    num = x + pad_lo + pad_hi - (dilation * (k - 1) + 1)
    q = abs(num) // stride
    return (q if num >= 0 else -q) + 1


class Operator:
    """Field handling of ts::Operator (src/runtime/operator.cpp:22-128)."""

    op = "operator"

    def __init__(self):
        self._fields = {}
        self._params = {}

    def field(self, name, attr, default=None):
        self._fields[name] = attr
        if default is not None:
            self._params[name] = default

    def has(self, name):
        return name in self._params

    def get(self, name):
        if name not in self._params:
            raise EjectionException('Unidentified param "%s"' % name)
        return self._params[name]

    def set(self, name, value):
        if name not in self._fields:
            raise EjectionException('Unidentified param "%s", did you mean "%s"' % (name, self._closest(name)))
        self._params[name] = value

    def _closest(self, name):
        import difflib
        m = difflib.get_close_matches(name, list(self._fields), n=1, cutoff=0.0)
        return m[0] if m else ""

    def init(self):
        missing = [f for f, a in self._fields.items() if a == REQUIRED and f not in self._params]
        if missing:
            raise EjectionException("Operator %s has unsatisfied fields: %s" % (self.op, ", ".join(missing)))


def _auto_check(cond, text):
    if not cond:
        raise EjectionException("Check failed: (%s)." % text)


class Quantize(Operator):
    """Operator "quantize" on the GPU: fp32 -> int8, attribute ``quantize_scale`` (one scale per sample)."""

    op = "quantize"

    def __init__(self):
        super().__init__()
        self.field("quantize_scale", REQUIRED)
        self.scales = None
        self._array = self._array_of = None

    def init(self):
        super().init()
        self.scales = [float(v) for v in np.asarray(self.get("quantize_scale"), dtype=np.float32).reshape(-1)]
        self._scale_array()

    def infer(self, inputs):
        _auto_check(len(inputs) == 1, "stack.size() == 1")
        x = inputs[0]
        _auto_check(len(self.scales) == x.shape[0], "m_quantize_scales.size() == x_tensor.sizes()[0]")
        return [("int8", tuple(x.shape))]

    def _scale_array(self):
        """The scales as the library takes them, laid out again when they are others than last time."""
        if self.scales != self._array_of:
            self._array, self._array_of = float_array(self.scales), list(self.scales)
        return self._array

    def run(self, inputs, stream=None):
        self.infer(inputs)
        x = inputs[0]
        if x.dtype not in (torch.float32, torch.float64):   # the reference's dispatch: src/kernels/cpu/quantize.cpp:130-141
            raise EjectionException("%s not support this data type: %s" % (self.op, str(x.dtype).replace("torch.", "")))
        x = x.contiguous()
        y = torch.empty(x.shape, dtype=torch.int8, device=x.device)
        lib = _lib.load()
        fn = lib.tsb_quantize_f32_i8 if x.dtype == torch.float32 else lib.tsb_quantize_f64_i8
        scales = self._scale_array()
        status = fn(x.data_ptr(), y.data_ptr(), x.numel(), scales, len(scales), _stream_ptr(stream))
        if status:
            check(status)
        return y


class Call:
    """A library call with every argument but the stream bound, and what those arguments point to kept alive: ``tensors``, and
    ``keep`` for the rest.

    ``sources``: (container, key, object) of the objects among them that a program could replace, for those who call again and again
    (BoundCalls)."""

    __slots__ = ("fn", "args", "keep", "tensors", "sources")

    def __init__(self, fn, args, keep, tensors, sources=()):
        self.fn, self.args, self.keep, self.tensors, self.sources = fn, args, keep, tensors, sources

    def __call__(self, stream_ptr):
        status = self.fn(*self.args, stream_ptr)
        if status:
            check(status)


class BoundCalls:
    """Calls that are made one after the other as long as they would be bound the same today: the containers that their objects came
    from still hold them, and every tensor still lies where it did.

    The check (some 0.7 us a call) goes ahead of the calls in groups, so that the GPU, which is busy with a call for longer than
    the host, does not wait for it."""

    GROUP = 6

    def __init__(self, calls):
        self.groups = []
        for i in range(0, len(calls), self.GROUP):
            group = calls[i:i + self.GROUP]
            containers, keys, held = zip(*[s for c in group for s in c.sources])
            where = [t.data_ptr for c in group for t in c.tensors if t is not None]
            self.groups.append((group, containers, keys, held, where, [f() for f in where]))

    def run(self, stream_ptr):
        """Makes the calls; False, with some of them made, once one would be bound differently."""
        for group, containers, keys, held, where, at in self.groups:
            try:
                if not all(map(operator.is_, map(operator.getitem, containers, keys), held)) or [f() for f in where] != at:
                    return False
            except (KeyError, IndexError):
                return False
            for call in group:
                status = call.fn(*call.args, stream_ptr)
                if status:
                    check(status)
        return True


def _scales_of(values):
    return values if isinstance(values, ctypes.Array) else float_array(values)


def _epilogue(dq, bias, residual, activation, leaky, out_f32, out_f32_layout, out_i8, out_i8_layout, requant_scales, out_acc,
              residual_after_activation):
    """The ConvEpilogue of these tensors (it refers to requant_scales, a ctypes array, which the caller keeps)."""
    e = ConvEpilogue()
    e.dequantize_scales = dq.data_ptr()
    e.activation = int(activation)
    e.leaky_scale = leaky
    if residual_after_activation:
        e.residual_after_activation = 1
    if bias is not None:
        e.bias = bias.data_ptr()
    if residual is not None:
        e.residual = residual.data_ptr()
    if out_f32 is not None:
        e.out_f32 = out_f32.data_ptr()
    e.out_f32_layout = out_f32_layout
    if out_i8 is not None:
        e.out_i8 = out_i8.data_ptr()
    e.out_i8_layout = out_i8_layout
    if requant_scales is not None:
        e.requant_scales_host = requant_scales
        e.n_requant_scales = len(requant_scales)
    if out_acc is not None:
        e.out_acc = out_acc.data_ptr()
    return e


class ConvPlan:
    """Owner of a tsb_conv_plan, its workspace and the device copies of the per-channel vectors."""

    def __init__(self, xshape, wshape, pad, stride, dilation, padding_value=0.0, kernel=KERNEL_AUTO, device="cuda",
                 mma_orientation=0, raw_row_mode=0, patch_mode=0):
        lib = self._lib = _lib.load()
        d = ConvDesc()
        d.mma_orientation, d.raw_row_mode, d.patch_mode = int(mma_orientation), int(raw_row_mode), int(patch_mode)
        d.n, d.c, d.h, d.w = [int(v) for v in xshape]
        d.o, _, d.kh, d.kw = [int(v) for v in wshape]
        d.pad_top, d.pad_bottom, d.pad_left, d.pad_right = [int(v) for v in pad]
        d.stride_h, d.stride_w = [int(v) for v in stride]
        d.dilation_h, d.dilation_w = [int(v) for v in dilation]
        d.padding_value = float(padding_value)
        d.kernel = int(kernel)
        self.desc = d
        handle = ctypes.c_void_p()
        check(lib.tsb_conv2d_i8_plan_create(ctypes.byref(d), ctypes.byref(handle)))
        self.handle = handle
        shape = (ctypes.c_int * 4)()
        check(lib.tsb_conv2d_i8_output_shape(handle, shape))
        self.out_shape = tuple(shape)
        self.kernel = lib.tsb_conv2d_i8_kernel(handle)
        self.ws_bytes = lib.tsb_conv2d_i8_workspace_bytes(handle)
        self.workspace = torch.empty(self.ws_bytes, dtype=torch.uint8, device=device)
        self.weights = None
        self.device = device

    def __del__(self):
        try:
            if self.handle:
                _lib.load().tsb_conv2d_i8_plan_destroy(self.handle)
                self.handle = None
        except Exception:
            pass

    def set_weights(self, w, stream=None):
        assert w.dtype == torch.int8 and w.is_cuda
        self.weights = w.contiguous()  # the direct kernel reads this tensor at run time
        check(_lib.load().tsb_conv2d_i8_set_weights(self.handle, _ptr(self.weights), _ptr(self.workspace), self.ws_bytes,
                                                    _stream_ptr(stream)))

    def quantize_input(self, x_f32, scales, stream=None):
        """fp32 NCHW -> the plan's staged int8 input; run() is then called with x=None, x_layout=LAYOUT_STAGED."""
        arr = scales if not isinstance(scales, (list, tuple)) else float_array(scales)
        status = self._lib.tsb_conv2d_i8_quantize_input(self.handle, x_f32.data_ptr(), arr, len(arr), self.workspace.data_ptr(),
                                                        self.ws_bytes, _stream_ptr(stream))
        if status:
            check(status)

    def run(self, x, x_layout, dq, bias=None, residual=None, activation=ACT_NONE, leaky=0.0, out_f32=None,
            out_f32_layout=LAYOUT_NCHW, out_i8=None, out_i8_layout=LAYOUT_NCHW, requant_scales=None, out_acc=None,
            stream=None, residual_after_activation=False):
        rq = None if requant_scales is None else _scales_of(requant_scales)
        e = _epilogue(dq, bias, residual, activation, leaky, out_f32, out_f32_layout, out_i8, out_i8_layout, rq, out_acc,
                      residual_after_activation)
        status = self._lib.tsb_conv2d_i8_run(self.handle, None if x is None else x.data_ptr(), x_layout, e, self.workspace.data_ptr(),
                                             self.ws_bytes, _stream_ptr(stream))
        if status:
            check(status)

    def bind_run(self, x, x_layout, dq, bias=None, residual=None, activation=ACT_NONE, leaky=0.0, out_f32=None,
                 out_f32_layout=LAYOUT_NCHW, out_i8=None, out_i8_layout=LAYOUT_NCHW, requant_scales=None,
                 residual_after_activation=False):
        """run() with these tensors as a Call, for programs that launch the same layer on the same buffers again and again."""
        rq = None if requant_scales is None else _scales_of(requant_scales)
        e = _epilogue(dq, bias, residual, activation, leaky, out_f32, out_f32_layout, out_i8, out_i8_layout, rq, None,
                      residual_after_activation)
        args = (self.handle, _ptr(x), int(x_layout), ctypes.byref(e), self.workspace.data_ptr(), self.ws_bytes)
        return Call(self._lib.tsb_conv2d_i8_run, args, (self, e, rq), (self.workspace, x, dq, bias, residual, out_f32, out_i8))

    def bind_projected(self, x, shortcut, x_shortcut, dq, shortcut_dq, bias=None, shortcut_bias=None, activation=ACT_NONE,
                       leaky=0.0, out_f32=None, out_i8=None, requant_scales=None, residual_after_activation=False,
                       tile_channels=0):
        """run_projected() with these tensors as a Call."""
        rq = None if requant_scales is None else _scales_of(requant_scales)
        e = _epilogue(dq, bias, None, activation, leaky, out_f32, LAYOUT_NHWC_PAD, out_i8, LAYOUT_NHWC_PAD, rq, None,
                      residual_after_activation)
        args = (self.handle, _ptr(x), shortcut.handle, _ptr(x_shortcut), _ptr(shortcut_dq), _ptr(shortcut_bias), ctypes.byref(e),
                int(tile_channels), self.workspace.data_ptr(), self.ws_bytes)
        return Call(self._lib.tsb_conv2d_i8_run_projected, args, (self, shortcut, e, rq),
                    (self.workspace, shortcut.workspace, x, x_shortcut, dq, shortcut_dq, bias, shortcut_bias, out_f32, out_i8))

    def run_projected(self, x, shortcut, x_shortcut, dq, shortcut_dq, bias=None, shortcut_bias=None, activation=ACT_NONE,
                      leaky=0.0, out_f32=None, out_i8=None, requant_scales=None, stream=None,
                      residual_after_activation=False, tile_channels=0):
        """This convolution with the 1x1 projection `shortcut` (another ConvPlan, its weights set) as its residual, in
        one launch (tsb_conv2d_i8_run_projected): NHWC_PAD int8 inputs, pixel-major fp32 / NHWC_PAD int8 outputs."""
        self.bind_projected(x, shortcut, x_shortcut, dq, shortcut_dq, bias, shortcut_bias, activation, leaky, out_f32, out_i8,
                            requant_scales, residual_after_activation, tile_channels)(_stream_ptr(stream))

    def bind_concat(self, x, first, x_first, dq, bias=None, activation=ACT_NONE, leaky=0.0, out_f32=None, out_i8=None,
                    requant_scales=None, tile_channels=0):
        """run_concat() with these tensors as a Call."""
        rq = None if requant_scales is None else _scales_of(requant_scales)
        e = _epilogue(dq, bias, None, activation, leaky, out_f32, LAYOUT_NHWC_PAD, out_i8, LAYOUT_NHWC_PAD, rq, None, False)
        args = (self.handle, _ptr(x), first.handle, _ptr(x_first), ctypes.byref(e), int(tile_channels), self.workspace.data_ptr(),
                self.ws_bytes)
        return Call(self._lib.tsb_conv2d_i8_run_concat, args, (self, first, e, rq),
                    (self.workspace, first.workspace, x, x_first, dq, bias, out_f32, out_i8))

    def run_concat(self, x, first, x_first, dq, bias=None, activation=ACT_NONE, leaky=0.0, out_f32=None, out_i8=None,
                   requant_scales=None, stream=None, tile_channels=0):
        """The convolution over concat(x_first, x) along channels in one launch (tsb_conv2d_i8_run_concat): `first` holds the
        weight columns of the leading channels (a 1x1 plan), this plan the rest; NHWC_PAD int8 inputs quantized with the
        same scales, pixel-major fp32 / NHWC_PAD int8 outputs."""
        self.bind_concat(x, first, x_first, dq, bias, activation, leaky, out_f32, out_i8, requant_scales,
                         tile_channels)(_stream_ptr(stream))

    def status(self, stream=None):
        check(_lib.load().tsb_conv2d_i8_status(self.handle, _ptr(self.workspace), _stream_ptr(stream)))

    def describe(self):
        buf = ctypes.create_string_buffer(512)
        n = _lib.load().tsb_conv2d_i8_plan_describe(self.handle, buf, len(buf))
        if n < 0:
            check(n)
        return buf.value.decode()


def _to_string(arr):
    return "[" + ", ".join(str(int(v)) for v in arr) + "]"


def _writes(t):
    """How often a tensor's memory was written so far; None where PyTorch does not count (inference tensors)."""
    return None if t.is_inference() else t._version


class Conv2DQuantized(Operator):
    """Operator "conv2d_quantized" on the GPU: int8 NCHW x int8 OIHW -> fp32 NCHW."""

    op = "conv2d_quantized"

    def __init__(self, kernel=KERNEL_AUTO):
        super().__init__()
        self.field("format", REQUIRED)
        self.field("padding", REQUIRED)
        self.field("padding_value", OPTIONAL, 0.0)
        self.field("stride", REQUIRED)
        self.field("dilation", OPTIONAL)
        self.field("dialations", OPTIONAL)
        self.field("dequantize_scales", REQUIRED)
        self._kernel = kernel
        # plans by what they were made from, this operator's own configuration included: attributes that are set again do not
        # meet a plan of the ones before them, and a plan that a captured graph refers to stays where it is
        self._plans = {}
        self._dq_dev = {}
        self._config = None

    def init(self):
        self._config = object()           # no plan is of a configuration that fails a check below
        super().init()
        fmt = self.get("format")
        padding = np.asarray(self.get("padding")).astype(np.int32)
        self.padding_value = float(np.asarray(self.get("padding_value")).reshape(-1)[0])
        stride = np.asarray(self.get("stride")).astype(np.int32)
        dilation = None
        if self.has("dilation"):
            dilation = np.asarray(self.get("dilation")).astype(np.int32)
        elif self.has("dialations"):
            dilation = np.asarray(self.get("dialations")).astype(np.int32)
        if dilation is None or dilation.size == 0:
            raise EjectionException("%s must set dilation or dialations" % self.op)
        _auto_check(padding.shape == (4, 2), "padding_tensor.has_shape({ 4, 2 })")
        _auto_check(stride.shape == (4,), "stride_tensor.has_shape({ 4, })")
        _auto_check(dilation.shape == (4,), "dilation_tensor.has_shape({ 4, })")
        if fmt not in ("NCHW", "NHWC"):
            raise EjectionException("%s do not support format: %s" % (self.op, fmt))
        self.format = fmt
        p = padding.reshape(-1)
        if fmt == "NCHW":
            bad_p, bad_s, bad_d = p[:4].any(), (stride[:2] != 1).any(), (dilation[:2] != 1).any()
        else:
            bad_p = p[[0, 1, 6, 7]].any()
            bad_s, bad_d = (stride[[0, 3]] != 1).any(), (dilation[[0, 3]] != 1).any()
        if bad_p:
            raise EjectionException("%s do not support padding: %s" % (self.op, _to_string(p)))
        if bad_s:
            raise EjectionException("%s do not support stride: %s" % (self.op, _to_string(stride)))
        if bad_d:
            raise EjectionException("%s do not support dialations: %s" % (self.op, _to_string(dilation)))
        self.padding4x2, self.stride4, self.dilation4 = p, stride, dilation
        self.dequantize_scales = np.asarray(self.get("dequantize_scales"), dtype=np.float32).reshape(-1)
        self._config = (fmt, p.tobytes(), stride.tobytes(), dilation.tobytes(), self.padding_value, self.dequantize_scales.tobytes())

    def _geometry(self):
        p, s, d = self.padding4x2, self.stride4, self.dilation4
        if self.format == "NCHW":
            return (p[4], p[5], p[6], p[7]), (s[2], s[3]), (d[2], d[3])
        return (p[2], p[3], p[4], p[5]), (s[1], s[2]), (d[1], d[2])

    def infer(self, inputs):
        _auto_check(len(inputs) == 2, "stack.size() == 2")
        x, w = inputs
        _auto_check(x.dim() == 4, "x_tensor.dims() == 4")
        _auto_check(w.dim() == 4, "w_tensor.dims() == 4")
        _auto_check(x.dtype == w.dtype, "x_tensor.dtype() == w_tensor.dtype()")
        _auto_check(w.shape[1] == x.shape[1], "w_tensor.size(1) == x_tensor.size(1)")
        _auto_check(x.dtype == torch.int8, "x_tensor.dtype() == INT8")
        _auto_check(len(self.dequantize_scales) == w.shape[0], "m_dequantize_scales.size() == w_tensor.size(0)")
        pad, stride, dil = self._geometry()
        if self.format == "NCHW":
            H, W, KH, KW = x.shape[2], x.shape[3], w.shape[2], w.shape[3]
        else:
            H, W, KH, KW = x.shape[1], x.shape[2], w.shape[1], w.shape[2]
        OH = conv_out_dim(H, pad[0], pad[1], KH, stride[0], dil[0])
        OW = conv_out_dim(W, pad[2], pad[3], KW, stride[1], dil[1])
        if self.format == "NCHW":
            return [("float32", (x.shape[0], w.shape[0], OH, OW))]
        return [("float32", (x.shape[0], OH, OW, w.shape[0]))]

    def run(self, inputs, stream=None, out_acc=None):
        """The weights are packed when they are new and when they were written since, as far as PyTorch counts writes (a write
        through ``.data`` or a raw pointer is not counted)."""
        kept = None
        if len(inputs) == 2:
            x, w = inputs
            # a plan was made for this configuration, these shapes and types only after they had passed every check
            key = (self._config, x.shape, w.shape, w.stride(), w.data_ptr(), x.dtype, w.dtype, x.device)
            kept = self._plans.get(key)
        if kept is None:
            self.infer(inputs)
            if self.format != "NCHW":
                raise EjectionException("Conv2D_quantized only support NCHW")  # conv2d_quantized_core.cpp:131-133
            pad, strides, dil = self._geometry()
            try:
                plan = ConvPlan(x.shape, w.shape, pad, strides, dil, self.padding_value, self._kernel, x.device)
            except TsbError as e:
                raise EjectionException(e.message)
            plan.set_weights(w, stream)
            # (the tensor is kept, so that its address stays its own)
            self._plans[key] = [plan, w, _writes(w)]
        else:
            plan = kept[0]
            writes = _writes(w)
            if writes is None or writes != kept[2]:
                plan.set_weights(w, stream)
                kept[2] = writes
        dq = self._dq_dev.get((self._config, x.device))
        if dq is None:
            dq = self._dq_dev[self._config, x.device] = torch.from_numpy(self.dequantize_scales.copy()).to(x.device)
        x = x.contiguous()
        out = torch.empty(plan.out_shape, dtype=torch.float32, device=x.device)
        plan.run(x, LAYOUT_NCHW, dq, out_f32=out, out_acc=out_acc, stream=stream)
        return out


def add_bias(x, bias, stream=None):
    """Operator "add_bias", format NCHW (src/kernels/gpu/add_bias.cu:19-26)."""
    x = x.contiguous()
    y = torch.empty_like(x)
    n, c = x.shape[0], x.shape[1]
    check(_lib.load().tsb_add_bias_f32_nchw(_ptr(x), _ptr(y), n, c, x.numel() // (n * c), _ptr(bias), _stream_ptr(stream)))
    return y


def relu(x, stream=None):
    x = x.contiguous()
    y = torch.empty_like(x)
    check(_lib.load().tsb_relu_f32(_ptr(x), _ptr(y), x.numel(), _stream_ptr(stream)))
    return y


def leaky_relu(x, scale, stream=None):
    x = x.contiguous()
    y = torch.empty_like(x)
    check(_lib.load().tsb_leaky_relu_f32(_ptr(x), _ptr(y), x.numel(), float(scale), _stream_ptr(stream)))
    return y


def quantize_nchw_to_nhwc(x, scales, stream=None):
    """fp32 NCHW -> int8 NHWC_PAD with the arithmetic of "quantize"."""
    x = x.contiguous()
    n, c, h, w = x.shape
    y = torch.empty((n, h, w, padded_channels(c)), dtype=torch.int8, device=x.device)
    check(_lib.load().tsb_quantize_f32_nchw_to_nhwc(_ptr(x), _ptr(y), n, c, h, w, float_array(scales), len(scales),
                                                    _stream_ptr(stream)))
    return y


def repack_nchw_to_nhwc(x, stream=None):
    x = x.contiguous()
    n, c, h, w = x.shape
    y = torch.empty((n, h, w, padded_channels(c)), dtype=torch.int8, device=x.device)
    check(_lib.load().tsb_repack_i8_nchw_to_nhwc(_ptr(x), _ptr(y), n, c, h, w, _stream_ptr(stream)))
    return y


def repack_nhwc_to_nchw(x, channels, stream=None):
    x = x.contiguous()
    n, h, w, _ = x.shape
    y = torch.empty((n, channels, h, w), dtype=torch.int8, device=x.device)
    check(_lib.load().tsb_repack_i8_nhwc_to_nchw(_ptr(x), _ptr(y), n, channels, h, w, _stream_ptr(stream)))
    return y
