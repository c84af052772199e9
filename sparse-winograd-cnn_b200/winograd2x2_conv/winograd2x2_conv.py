"""Drop-in for the reference module of the same path (winograd2x2_cublas/winograd2x2_conv/
winograd2x2_conv.py:13-36): same function names and tensor shapes, on torch CUDA tensors.

    winograd2x2_conv(I, W)              I (16,B,nH,nW,C), W (16,C,K) -> (B,2nH,2nW,K); differentiable
    winograd2x2_conv_grad(i1, i2, grad) -> (grad wrt I, grad wrt W)

`math` selects the FP32 FFMA kernels ("fp32") or the tcgen05 TF32 kernels ("tf32");
`out_hw` crops the output to odd image sizes; `data_format="NCHW"` is an extension.
"""
from wg2x2 import ops as _ops


def winograd2x2_conv(I, W, out_hw=None, data_format="NHWC", math="fp32", mask=None):
    """mask: a constant pruning mask of W's shape; the product is that of I and W * mask."""
    oh, ow = out_hw if out_hw is not None else (None, None)
    return _ops.conv_op(I, W, oh, ow, data_format, math, mask)


def winograd2x2_conv_grad(i1, i2, grad, data_format="NHWC", math="fp32"):
    return _ops.conv_bwd(i1.contiguous(), i2.contiguous(), grad.contiguous(), layout=data_format, math=math)
