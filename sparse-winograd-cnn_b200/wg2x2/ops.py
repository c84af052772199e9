"""Torch-facing calls into the C ABI: device memory and streams come from PyTorch, the
arithmetic is entirely in libwinograd2x2_b200.so.  The work of a call (argument checks, allocation, stream lookup,
launch) is native code, csrc/bindings.cpp; the functions here give it names, keywords and defaults."""
import torch

from . import _lib
from ._lib import MATH_FP32, MATH_TF32, NCHW, NHWC, Wg2x2Error, lib
from . import _native

_native.set_error(Wg2x2Error)

_LAYOUTS = {"NHWC": NHWC, "NCHW": NCHW, NHWC: NHWC, NCHW: NCHW}
_MATHS = {"fp32": MATH_FP32, "tf32": MATH_TF32, MATH_FP32: MATH_FP32, MATH_TF32: MATH_TF32}


def _chk(t, name):
    if not (isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == torch.float32 and t.is_contiguous()):
        raise TypeError("%s must be a contiguous float32 CUDA tensor" % name)
    return t


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ptr(t):
    return None if t is None else t.data_ptr()


def imtrans_fwd(x, relu=False, layout="NHWC", out=None, in_scale=None, in_shift=None):
    """x (B,H,W,C) or (B,C,H,W) -> V (16,B,nH,nW,C); in_scale/in_shift (C,) apply x*scale+shift to the pixels first."""
    return _native.imtrans_fwd(x, relu, _LAYOUTS[layout], out, in_scale, in_shift)


def imtrans_bwd(dV, H, W, V_relu=None, layout="NHWC"):
    """dV (16,B,nH,nW,C) -> dX; V_relu, if given, applies the ReLU mask V>0 first."""
    return _native.imtrans_bwd(dV, H, W, V_relu, _LAYOUTS[layout])


class _ImTransTraced(torch.autograd.Function):
    """imtrans_op in the form that torch.jit.trace records, a Python operator; the native calls it does not see.  (The outputs come
    from torch: the tracer wants to know where a tensor with gradients is from.)"""

    @staticmethod
    def forward(ctx, x, relu, layout):
        B, H, W, C = (int(n) for n in (x.shape if layout == NHWC else (x.shape[0], x.shape[2], x.shape[3], x.shape[1])))
        V = imtrans_fwd(x.contiguous(), relu, layout, out=x.new_empty((16, B, (H + 1) // 2, (W + 1) // 2, C)))
        ctx.hw = H, W
        ctx.layout, ctx.relu = layout, relu
        if relu:
            ctx.save_for_backward(V)
        return V

    @staticmethod
    def backward(ctx, g):
        V = ctx.saved_tensors[0] if ctx.relu else None
        return imtrans_bwd(g.contiguous(), ctx.hw[0], ctx.hw[1], V, ctx.layout), None, None


class _ConvTraced(torch.autograd.Function):
    """conv_op likewise, without the mask."""

    @staticmethod
    def forward(ctx, V, Wt, out_h, out_w, layout, math):
        V, Wt = V.contiguous(), Wt.contiguous()
        ctx.save_for_backward(V, Wt)
        ctx.layout, ctx.math = layout, math
        B, nH, nW, K = (int(n) for n in (*V.shape[1:4], Wt.shape[2]))
        H, W = 2 * nH if out_h is None else out_h, 2 * nW if out_w is None else out_w
        return conv_fwd(V, Wt, H, W, layout, math, out=V.new_empty((B, H, W, K) if layout == NHWC else (B, K, H, W)))

    @staticmethod
    def backward(ctx, g):
        V, Wt = ctx.saved_tensors
        dV, dW = conv_bwd(V, Wt, g.contiguous(), layout=ctx.layout, math=ctx.math, need_dV=ctx.needs_input_grad[0], need_dW=ctx.needs_input_grad[1])
        return dV, dW, None, None, None, None


def imtrans_op(x, relu=False, layout="NHWC"):
    """imtrans_fwd for autograd: differentiable in x (any strides), the ReLU mask applied inside the gradient's gather."""
    V = _native.imtrans_op(x, relu, _LAYOUTS[layout])
    return V if V is not NotImplemented else _ImTransTraced.apply(x, bool(relu), _LAYOUTS[layout])


def conv_fwd(V, Wt, out_h=None, out_w=None, layout="NHWC", math="fp32", out=None, workspace=None):
    """V (16,B,nH,nW,C), Wt (16,C,K) -> Y (B,out_h,out_w,K) / (B,K,out_h,out_w)."""
    return _native.conv_fwd(V, Wt, out_h, out_w, _LAYOUTS[layout], _MATHS[math], out, workspace)


def conv_op(V, Wt, out_h=None, out_w=None, layout="NHWC", math="fp32", mask=None):
    """conv_fwd for autograd: differentiable in V and Wt (any strides).  mask (16,C,K), constant: the weights are Wt * mask."""
    Y = _native.conv_op(V, Wt, out_h, out_w, _LAYOUTS[layout], _MATHS[math], mask)
    if Y is NotImplemented:
        out_hw = (None if n is None else int(n) for n in (out_h, out_w))
        Y = _ConvTraced.apply(V, Wt if mask is None else Wt * mask, *out_hw, _LAYOUTS[layout], _MATHS[math])
    return Y


def prepare_weights(Wt):
    """Wt (16,C,K) -> opaque device buffer for conv_fwd_prepared (TF32 tensor-core path)."""
    _chk(Wt, "Wt")
    _, C, K = Wt.shape
    n = lib.wg2x2_prepared_weights_bytes(C, K)
    buf = torch.empty(n, dtype=torch.uint8, device=Wt.device)
    with torch.cuda.device(Wt.device):
        _lib.check(lib.wg2x2_weights_prepare(_ptr(Wt), C, K, _ptr(buf), n, _stream()), "wg2x2_weights_prepare")
    buf._wg_ck = (C, K)
    return buf


def conv_fwd_prepared(V, prepared, K, out_h=None, out_w=None, layout="NHWC", out=None, out_scale=None, out_shift=None,
                      residual=None, workspace=None, wide=True):
    """As conv_fwd(math="tf32") with weights already prepared by prepare_weights; optionally
    Y = acc*out_scale[k] + out_shift[k] + residual in the kernel's epilogue."""
    return _native.conv_fwd_prepared(V, prepared, K, out_h, out_w, _LAYOUTS[layout], out, out_scale, out_shift, residual, workspace, wide)


def conv_bwd(V, Wt, dY, mask=None, layout="NHWC", relu=False, math="fp32", need_dV=True, need_dW=True):
    """Gradients (dV, dW) of conv_fwd for dY (B,H,W,K) / (B,K,H,W)."""
    return _native.conv_bwd(V, Wt, dY, mask, _LAYOUTS[layout], relu, _MATHS[math], need_dV, need_dW)


def layer_fwd(x, Wt, relu=True, layout="NHWC", math="fp32", keep_V=False, out=None, workspace=None):
    """Whole Winograd-ReLU layer X -> Y (and V when keep_V)."""
    return _native.layer_fwd(x, Wt, relu, _LAYOUTS[layout], _MATHS[math], keep_V, out, workspace)


def fused_supported(B, H, W, C, K, layout="NCHW"):
    return bool(lib.wg2x2_layer_fwd_fused_supported(B, H, W, C, K, _LAYOUTS[layout]))


def fused_preferred(B, H, W, C, K, layout="NCHW"):
    """True where the one-kernel NCHW layer (layer_fwd_fused) is preferred to transform and product as kernels of their own and to the
    layer on clusters, as for few tiles.  (Many tiles go to the layer on pairs of SMs before that is asked.)"""
    return bool(lib.wg2x2_layer_fwd_fused_preferred(B, H, W, C, K, _LAYOUTS[layout]))


def layer_fwd_prepared(x, prepared, K, relu=True, layout="NHWC", out=None, V_scratch=None, out_scale=None, out_shift=None,
                       residual=None, workspace=None, in_scale=None, in_shift=None, residual_relu=False):
    """Whole layer with prepared weights: one kernel where supported and faster (V never stored: kernels of their own for few
    and for many tiles, an NCHW one for few channels), else transform + product through V_scratch (allocated here when not given); layers
    with many channels take the wide product path through `workspace` (allocated here when not given;
    layer_fwd_prepared_workspace_bytes).  in_scale / in_shift (C,): affine map of the pixels in front of the transform, the
    padding stays zero; residual_relu: the shortcut passes through a ReLU first."""
    return _native.layer_fwd_prepared(x, prepared, K, relu, _LAYOUTS[layout], out, V_scratch, out_scale, out_shift, residual, workspace,
                                      in_scale, in_shift, residual_relu)


def layer_fwd_prepared_workspace_bytes(B, H, W, C, K):
    return int(lib.wg2x2_layer_fwd_prepared_workspace_bytes(B, H, W, C, K))


def layer_fwd_fused(x, prepared, K, relu=True, out=None, out_scale=None, out_shift=None, residual=None,
                    in_scale=None, in_shift=None):
    """The one-kernel layer forward (NCHW); raises Wg2x2Error(UNSUPPORTED) for other shapes.  in_scale/in_shift:
    per-input-channel affine map applied to the image in front of the transform (the padding stays zero)."""
    return _native.layer_fwd_fused(x, prepared, K, relu, out, out_scale, out_shift, residual, in_scale, in_shift)


def residual_block(x, shortcut, prepared_a, bn_a, prepared_b, bn_b, bn_out, K, layout="NCHW"):
    """shortcut + bn_out(layer_b(bn_b(layer_a(bn_a(x))))), both layers with prepared weights and K output channels; bn_*: (scale,
    shift) pairs.  The result is written over `shortcut`; with None the shortcut is relu(x)."""
    return _native.residual_block(x, shortcut, K, prepared_a, bn_a[0], bn_a[1], prepared_b, bn_b[0], bn_b[1], bn_out[0], bn_out[1],
                                  _LAYOUTS[layout])


def conv1x1(x, w):
    """1x1 convolution of x (B,C,H,W) with w (K,C,1,1), whose values have to be rounded to TF32 (round_tf32): (B,K,H,W), or None
    where the library's convolution is the better choice (many pixels; more than 256 channels)."""
    return _native.conv1x1(x, w)


def round_tf32(t):
    """t rounded to TF32, nearest with ties away from zero; NaN stays NaN."""
    t = t.contiguous()
    return torch.where(t.isnan(), t.new_tensor(float("nan")), ((t.view(torch.int32) + 0x1000) & ~0x1FFF).view(torch.float32))


def relu_mean(x):
    """x (B,C,H,W) -> (B,C): the mean of relu(x) over the pixels."""
    return _native.relu_mean(x)


def maxpool3x3s2_same(x, with_relu=False, relu_scale=None, relu_shift=None):
    """3x3 / stride 2 max-pooling with TensorFlow's SAME padding of a (B,C,H,W) tensor into NCHW outputs; with_relu=True
    returns (pooled, relu(relu_scale[c] * pooled + relu_shift[c])) from the same pass (scale 1, shift 0 when not given).
    x may be contiguous (NCHW) or channels-last (e.g. the output of a channels-last convolution)."""
    return _native.maxpool(x, with_relu, relu_scale, relu_shift)


def stem_supported(H, W):
    """Image sizes the fused 7x7/2 convolution + pool kernel takes: multiples of 4, at most 224 wide."""
    return H >= 4 and W >= 4 and H % 4 == 0 and W % 4 == 0 and W <= 224


def stem_prepare(w):
    """(64,3,7,7) stem weights -> the arrangement stem7x7s2_pool reads (TF32-rounded, in fragment order)."""
    _chk(w, "w")
    if tuple(w.shape) != (64, 3, 7, 7):
        raise ValueError("stem weights must have shape (64,3,7,7), got %s" % (tuple(w.shape),))
    wp = torch.empty(lib.wg2x2_stem_prepared_floats(), dtype=torch.float32, device=w.device)
    with torch.cuda.device(w.device):
        _lib.check(lib.wg2x2_stem_prepare(_ptr(w), _ptr(wp), _stream()), "wg2x2_stem_prepare")
    return wp


def stem7x7s2_pool(x, prepared, with_relu=False, relu_scale=None, relu_shift=None):
    """pool1(conv1(x)) of the ResNet-18-var graph in one kernel: x (B,3,H,W) -> (B,64,H/4,W/4); with_relu=True also
    returns relu(relu_scale[c] * pooled + relu_shift[c]).  `prepared` comes from stem_prepare."""
    _chk(x, "x")
    B, C, H, W = x.shape
    if C != 3:
        raise ValueError("stem input must have 3 channels, got %d" % C)
    if not stem_supported(H, W):
        raise ValueError("stem kernel needs H and W multiples of 4 and W <= 224, got %dx%d" % (H, W))
    return _native.stem_pool(x, prepared, with_relu, relu_scale, relu_shift)


def last_device_status():
    """(status, where) of the bounded device-side waits since the last reading; synchronises the current stream.
    The tensor-core calls above do not read it themselves (that would cost a synchronisation per call): after a
    time-out their outputs are incomplete, so a caller that must know polls here after its last launch."""
    import ctypes
    where = ctypes.c_uint(0)
    st = lib.wg2x2_last_device_status(_stream(), ctypes.byref(where))
    return st, where.value
