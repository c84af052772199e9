"""The work whose speed counts: cases over the range of sizes, layouts, precisions and directions that users of this
library run, each through the public Python entry points.

`listed()` names twelve cases, `draw(rng)` gives further ones of the same ranges; `prepare`, `run`, `work` and `tolerance`
take a case.  Kinds:

  layer    inference of one Winograd-ReLU layer with prepared weights (tensor cores): wg2x2.layer_fwd_prepared, plain or as
           the end of a residual block (folded BatchNorm and shortcut)
  forward  the layer wrappers without gradients: WinogradImTrans(relu) + WinogradConvLayer, in their default precision
  train    the layer wrappers with gradients: forward, then dX and dW, as one layer of a training step
  grad     the gradient calls on their own, with the pruning mask and the ReLU mask in the product's epilogue
  net      the ResNet-18-var forward pass on a batch of 224 x 224 images
"""
import functools
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("sparse-winograd-cnn_b200"))

import resnet18_var  # noqa: E402
import wg2x2  # noqa: E402
import winograd_conv  # noqa: E402
import winograd_imtrans  # noqa: E402


def _layer(name, B, C, K, H, W, layout="NCHW", density=1.0, block_end=False):
    return dict(name=name, kind="layer", math="tf32", layout=layout, B=B, C=C, K=K, H=H, W=W, density=density, block_end=block_end)


def _wrapped(name, kind, math_mode, layout, B, C, K, H, W, density=1.0):
    return dict(name=name, kind=kind, math=math_mode, layout=layout, B=B, C=C, K=K, H=H, W=W, density=density)


def listed():
    return [
        # one image at a time: a conv2_x layer in a latency-bound service
        _layer("layer_1x64x56", 1, 64, 64, 56, 56),
        # the conv2_x layer at a throughput batch (the benchmark's headline workload)
        _layer("layer_64x64x56", 64, 64, 64, 56, 56),
        # the pruned conv4_x layer (benchmark workload cfg3): many channels, small image
        _layer("layer_128x256x14", 128, 256, 256, 14, 14, density=0.3),
        # odd image, channel counts off the tile sizes, end of a residual block: what a network that is not ResNet-shaped gives
        _layer("layer_ragged_5x48x27", 5, 48, 80, 27, 27, density=0.6, block_end=True),
        # the reference's own layout: channels last
        _layer("layer_nhwc_32x128x28", 32, 128, 128, 28, 28, layout="NHWC", density=0.4),
        # the reference's modules swapped for ours and nothing else changed: channels last, FP32, inference
        _wrapped("forward_fp32_8x256x14", "forward", "fp32", "NHWC", 8, 256, 256, 14, 14),
        # the same in training
        _wrapped("train_fp32_16x128x28", "train", "fp32", "NHWC", 16, 128, 128, 28, 28),
        # training a conv2_x layer on the tensor cores, the reference's layout
        _wrapped("train_nhwc_64x64x56", "train", "tf32", "NHWC", 64, 64, 64, 56, 56),
        # fine-tuning a pruned layer of a small ragged network: launches and host work count
        _wrapped("train_ragged_6x96x13", "train", "tf32", "NCHW", 6, 96, 72, 13, 15, density=0.5),
        # the conv5_x gradients of a large training batch (benchmark workload cfg5)
        _wrapped("grad_256x512x7", "grad", "tf32", "NCHW", 256, 512, 512, 7, 7, density=0.2),
        # the network: one image, and the benchmark's batch (cfg4)
        dict(name="net_1", kind="net", B=1),
        dict(name="net_256", kind="net", B=256),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# A drawn case stays below the largest listed one: bytes of the transformed input, and operations by precision
_MOST_V_BYTES = 260e6
_MOST_FLOPS = {"tf32": 70e9, "fp32": 20e9}


def draw(rng):
    kind = rng.choices(["layer", "forward", "train", "grad", "net"], [40, 10, 28, 10, 12])[0]
    if kind == "net":
        return dict(kind="net", B=_log_int(rng, 1, 256))
    math_mode = "fp32" if kind == "forward" or (kind == "train" and rng.random() < 0.4) else "tf32"
    layout = "NHWC" if math_mode == "fp32" else rng.choice(["NCHW", "NCHW", "NHWC"])
    while True:
        H = _log_int(rng, 7, 64)
        W = H if rng.random() < 0.7 else _log_int(rng, 7, 64)
        if kind == "layer" and rng.random() < 0.5:      # images of networks that halve 224 or 256 are multiples of 4
            H, W = -(-H // 4) * 4, -(-W // 4) * 4
        # channel counts: powers of two and their neighbours in steps of 16 or 4, about as many out as in
        step = rng.choice([64, 32, 16, 4])
        C = -(-_log_int(rng, 16, 512) // step) * step
        K = C if rng.random() < 0.6 else -(-_log_int(rng, 16, 512) // step) * step
        B = _log_int(rng, 1, 256)
        P = B * ((H + 1) // 2) * ((W + 1) // 2)
        flops = (1 if kind in ("layer", "forward") else 2 if kind == "grad" else 3) * 32.0 * P * C * K
        if 64.0 * P * max(C, K) <= _MOST_V_BYTES and flops <= _MOST_FLOPS[math_mode]:
            break
    density = rng.choice([1.0, 1.0, 0.6, 0.4, 0.3, 0.2])
    case = dict(kind=kind, math=math_mode, layout=layout, B=B, C=C, K=K, H=H, W=W, density=density)
    if kind == "layer":
        case["block_end"] = rng.random() < 0.3
    return case


@functools.lru_cache(maxsize=1)
def _network():
    """The network a program keeps; its weights do not depend on the images."""
    return resnet18_var.ResNet18Var().cuda().eval()


def _image(case, ch, gen):
    B, H, W = case["B"], case["H"], case["W"]
    shape = (B, ch, H, W) if case["layout"] == "NCHW" else (B, H, W, ch)
    return torch.randn(shape, generator=gen, device="cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(case)
    if case["kind"] == "net":
        s["model"] = _network()
        s["x"] = torch.randn((case["B"], 3, 224, 224), generator=gen, device="cuda")
        return s
    C, K, H, W, layout = case["C"], case["K"], case["H"], case["W"], case["layout"]
    s["x"] = _image(case, C, gen)
    # Winograd-domain weights at the reference's initialiser scale, pruned to the case's density
    w = torch.randn((16, C, K), generator=gen, device="cuda") * (1.3 * (2.0 * 9.0 / 32.0) / (16 * C)) ** 0.5
    mask = (torch.rand((16, C, K), generator=gen, device="cuda") < case["density"]).float() if case["density"] < 1.0 else None
    if case["kind"] == "layer":
        s["prepared"] = wg2x2.prepare_weights(w if mask is None else w * mask)
        s["extras"] = {}
        if case["block_end"]:
            s["extras"] = dict(out_scale=1.0 + 0.1 * torch.randn(K, generator=gen, device="cuda"),
                               out_shift=0.1 * torch.randn(K, generator=gen, device="cuda"), residual=torch.relu(_image(case, K, gen)))
    elif case["kind"] == "grad":
        s["mask"] = mask
        s["w"] = w if mask is None else w * mask
        s["v"] = wg2x2.imtrans_fwd(s["x"], relu=True, layout=layout)
        s["dy"] = _image(case, K, gen)
        del s["x"]
    else:
        s["layer"] = winograd_conv.WinogradConvLayer(C, K, mask=mask, W_init=lambda shape: w, device="cuda")
        if case["kind"] == "train":
            s["x"].requires_grad_(True)
            s["dy"] = _image(case, K, gen)
    return s


def _wrappers(s):
    v = winograd_imtrans.WinogradImTrans(s["x"], nl=torch.relu, data_format=s["layout"])
    return s["layer"](v, out_hw=(s["H"], s["W"]), data_format=s["layout"], math=s["math"])


def run(s):
    kind = s["kind"]
    if kind == "net":
        with torch.no_grad():
            return s["model"](s["x"])
    if kind == "layer":
        return wg2x2.layer_fwd_prepared(s["x"], s["prepared"], s["K"], relu=True, layout=s["layout"], **s["extras"])
    if kind == "forward":
        with torch.no_grad():
            return _wrappers(s)
    if kind == "train":
        y = _wrappers(s)
        dx, dw = torch.autograd.grad(y, (s["x"], s["layer"].W), s["dy"])
        return y.detach(), dx, dw
    dv, dw = wg2x2.conv_bwd(s["v"], s["w"], s["dy"], mask=s["mask"], layout=s["layout"], relu=True, math=s["math"])
    return wg2x2.imtrans_bwd(dv, s["H"], s["W"], layout=s["layout"]), dw


def work(case):
    """Bytes: every input read once, every output written once.  Operations: the dense products."""
    B = case["B"]
    if case["kind"] == "net":
        weights = 3 * 49 * 64 + 512 * 1000
        flops = 2.0 * B * (112 * 112 * 64 * 147 + 512 * 1000)
        for (cin, cout), side in zip(resnet18_var.STAGES, (56, 28, 14, 7)):
            tiles = B * ((side + 1) // 2) ** 2
            weights += 16 * (cin * cout + 3 * cout * cout) + cin * cout
            flops += 32.0 * tiles * (cin * cout + 3 * cout * cout) + 2.0 * B * side * side * cin * cout
        return dict(bytes=4.0 * (B * 3 * 224 * 224 + weights + B * 1000), flops=flops)
    C, K, H, W = case["C"], case["K"], case["H"], case["W"]
    P = B * ((H + 1) // 2) * ((W + 1) // 2)
    x, y, w, product = B * C * H * W, B * K * H * W, 16 * C * K, 32.0 * P * C * K
    masked = w if case["density"] < 1.0 else 0
    if case["kind"] == "layer":
        return dict(bytes=4.0 * (x + w + y + (y + 2 * K if case["block_end"] else 0)), flops=product)
    if case["kind"] == "forward":
        return dict(bytes=4.0 * (x + w + masked + y), flops=product)
    if case["kind"] == "train":      # X, W, mask, dY in; Y, dX, dW out
        return dict(bytes=4.0 * (x + w + masked + y + y + x + w), flops=3 * product)
    return dict(bytes=4.0 * (16 * P * C + w + masked + y + x + w), flops=2 * product)      # V, W, mask, dY in; dX, dW out


def tolerance(case):
    if case["kind"] == "net":        # TF32 products (11-bit operands, FP32 sums) through twenty layers
        return {"rel": 5e-3}
    if case["math"] == "tf32":       # one TF32 product, operands rounded or cut to 11 bits
        return {"rel": 2e-3}
    return {"rel": 1e-5}
