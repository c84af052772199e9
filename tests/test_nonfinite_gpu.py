"""NaN and infinity through the kernels that round operands to TF32 themselves or apply a ReLU of the network: where an operand is not
finite the result is not, as with cvt.rna.tf32, which the other kernels of the same step use, and torch.relu, which keeps NaN."""
import pytest
import torch
import torch.nn.functional as F

NANS = [0x7FFFFFFF, -1, 0x7FC00000, 0xFFC00000 - (1 << 32), 0x7F800001]     # CUDA's, all ones, the x86 pair, a payload in the low bits only


def _put(t, at, bits):
    t.view(torch.int32)[at] = bits


def _dm(dY):
    """A dY A^T in float64 by the additions of the kernels (a zero coefficient is no operand): (16, B, nH, nW, K) of dY (B, K, H, W)."""
    B, K, H, W = dY.shape
    g = F.pad(dY.double(), (0, W % 2, 0, H % 2)).reshape(B, K, (H + 1) // 2, 2, (W + 1) // 2, 2)
    ends = lambda a, b: [a, a + b, a - b, -b]
    return torch.stack([m for u0, u1 in zip(ends(g[:, :, :, 0, :, 0], g[:, :, :, 1, :, 0]), ends(g[:, :, :, 0, :, 1], g[:, :, :, 1, :, 1]))
                        for m in ends(u0, u1)]).permute(0, 1, 3, 4, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["NCHW", "NHWC"])
@pytest.mark.parametrize("shape", [(44, 32, 64, 14, 14), (90, 32, 128, 7, 7), (2, 32, 64, 14, 14)])      # two channels per lane twice, segments
def test_dy_reaches_the_gradients(shape, layout):
    import wg2x2
    B, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    v, w, clean = rnd(16, B, (H + 1) // 2, (W + 1) // 2, C), rnd(16, C, K), rnd(B, K, H, W)
    cases = [{(1, 3 + i, 5, 6 - i): n} for i, n in enumerate(NANS)]
    cases.append({(0, 2, 2, 4): 0x7F800000, (0, 2, 3, 4): 0x7F800000})              # inf - inf inside a tile
    cases.append({(1, 5, H - 1, W - 1): 0xFF800000 - (1 << 32)})
    for case in cases:
        dy = clean.clone()
        for at, bits in case.items():
            _put(dy, at, bits)
        dm = _dm(dy)
        dv, dw = wg2x2.conv_bwd(v, w, dy if layout == "NCHW" else dy.permute(0, 2, 3, 1).contiguous(), layout=layout, math="tf32")
        assert not dm.isfinite().all()
        assert torch.equal(~dv.isfinite(), (~dm.isfinite()).any(-1, keepdim=True).expand_as(dv))
        assert torch.equal(~dw.isfinite(), (~dm.isfinite()).any(3).any(2).any(1)[:, None, :].expand_as(dw))
        assert dv[dm.isnan().any(-1)].isnan().all() and dw.transpose(1, 2)[dm.isnan().any(3).any(2).any(1)].isnan().all()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 64, 48), (3, 224, 224)])
def test_image_reaches_the_stem(shape):
    """The kernel's eighth tap has weight zero, so a NaN reaches the outputs of 7 x 8 taps; the pool drops NaN beside a number."""
    import wg2x2
    from resnet18_var import _same_pool
    B, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(B + H + W)
    x, w = torch.randn((B, 3, H, W), device="cuda", generator=g), torch.randn((64, 3, 7, 7), device="cuda", generator=g) * 0.1
    prep = wg2x2.stem_prepare(w)
    for i, bits in enumerate(NANS):
        bad = x.clone()
        for c, y, z in ((i % 3, 10 + i, 11), (1, 0, 0), (2, H - 1, W - 1 - i)):
            bad[B - 1, c, y, z] = 0.0
        zero = bad.clone()
        for c, y, z in ((i % 3, 10 + i, 11), (1, 0, 0), (2, H - 1, W - 1 - i)):
            _put(bad, (B - 1, c, y, z), bits)
        nan = F.conv2d(F.pad(bad.isnan().float(), (2, 4, 2, 3)), torch.ones((1, 3, 7, 8), device="cuda"), stride=2) > 0.5
        conv = F.conv2d(F.pad(wg2x2.round_tf32(zero).double(), (2, 3, 2, 3)), wg2x2.round_tf32(w).double(), stride=2).float()
        want = _same_pool(conv.masked_fill(nan, float("-inf")))
        lost = torch.isneginf(want)
        assert lost.any()
        got = wg2x2.stem7x7s2_pool(bad, prep)
        assert torch.equal(got.isnan(), lost)
        assert float((got - want)[~lost].abs().max()) <= 2e-5 * float(want[~lost].abs().max())       # FP32 sums in another order


@pytest.mark.gpu
def test_image_and_weights_reach_the_1x1_convolution():
    import wg2x2
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.randn((2, 100, 9, 13), device="cuda", generator=g), torch.randn((70, 100, 1, 1), device="cuda", generator=g)
    for bits in NANS + [0x7F800000, 0xFF800000 - (1 << 32)]:
        bad, wbad = x.clone(), w.clone()
        _put(bad, (1, 37, 4, 5), bits)
        _put(wbad, (69, 2, 0, 0), bits)
        y, clean = wg2x2.conv1x1(bad, wg2x2.round_tf32(w)), wg2x2.conv1x1(x, wg2x2.round_tf32(w))
        hit = torch.zeros_like(y, dtype=torch.bool)
        hit[1, :, 4, 5] = True
        assert torch.equal(~y.isfinite(), hit) and torch.equal(y[~hit], clean[~hit])
        y = wg2x2.conv1x1(x, wg2x2.round_tf32(wbad))
        assert not y[:, 69].isfinite().any() and torch.equal(y[:, :69], clean[:, :69])


def test_round_tf32_values():
    """Nearest, ties away from zero, on any device; infinities stay, NaN stays NaN, what rounds beyond the largest value is infinite."""
    import wg2x2
    f = lambda *bits: torch.tensor([b - (1 << 32) if b >= 1 << 31 else b for b in bits], dtype=torch.int64).to(torch.int32).view(torch.float32)
    x = f(0x3F800FFF, 0x3F801000, 0xBF801000, 0x3F803000, 0x7F7FFFFF, 0x7F800000, 0xFF800000, 0x00000000, 0x80000000, 0x00001000)
    want = f(0x3F800000, 0x3F802000, 0xBF802000, 0x3F804000, 0x7F800000, 0x7F800000, 0xFF800000, 0x00000000, 0x80000000, 0x00002000)
    assert torch.equal(wg2x2.round_tf32(x).view(torch.int32), want.view(torch.int32))
    nans = f(*(n & 0xFFFFFFFF for n in NANS))
    assert wg2x2.round_tf32(nans).isnan().all()


# every kernel that adds relu(shortcut): few tiles (NCHW of even and odd width, NHWC with and without whole groups of four channels), the
# one-kernel layer, the wide path's output transforms, the row-walk kernel (NHWC in whole blocks and not, NCHW), the layer on pairs of SMs
# (in front of the stores: rows of 8- and 4-byte pieces, channels last, one unit a pair; behind them)
@pytest.mark.gpu
@pytest.mark.parametrize("shape,layout,kernel", [
    ((1, 56, 56, 64, 64), "NCHW", "clusters"), ((2, 9, 13, 32, 36), "NCHW", "clusters"), ((2, 9, 13, 32, 36), "NHWC", "clusters"), ((7, 7, 7, 128, 130), "NHWC", "clusters"),
    ((16, 56, 56, 64, 64), "NCHW", "one"), ((24, 14, 14, 256, 256), "NCHW", "wide"), ((48, 14, 14, 256, 256), "NHWC", "wide"), ((12, 13, 15, 256, 264), "NCHW", "wide"),
    ((24, 48, 46, 64, 64), "NHWC", "walk"), ((24, 48, 48, 64, 66), "NHWC", "walk"), ((40, 49, 49, 32, 64), "NCHW", "walk"),
    ((48, 14, 14, 256, 256), "NCHW", "pairs"), ((65, 27, 27, 96, 96), "NCHW", "pairs"), ((24, 48, 48, 64, 64), "NHWC", "pairs"), ((16, 40, 36, 96, 96), "NCHW", "pairs"),
    ((64, 56, 56, 64, 64), "NCHW", "pairs")])
def test_shortcut_reaches_the_output(shape, layout, kernel):
    import wg2x2
    from conftest import kernel_of
    assert kernel_of(*shape, layout, shortcut=1) == kernel
    B, H, W, C, K = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, r = (rnd(B, H, W, c) if layout == "NHWC" else rnd(B, c, H, W) for c in (C, K))
    flat = r.view(-1)
    for i, bits in enumerate(NANS + [0x7F800000, 0xFF800000 - (1 << 32)]):
        _put(flat, (flat.numel() // 9 * (i + 1) + i,), bits)
    prepared = wg2x2.prepare_weights(rnd(16, C, K) / C ** 0.5)
    kw = dict(relu=True, layout=layout, out_scale=1 + 0.2 * rnd(K), out_shift=0.3 * rnd(K))
    got = wg2x2.layer_fwd_prepared(x, prepared, K, residual=r, residual_relu=True, **kw)
    want = wg2x2.layer_fwd_prepared(x, prepared, K, residual=torch.relu(r), **kw)
    assert int(want.isnan().sum()) == len(NANS) and torch.equal(got.isnan(), want.isnan())
    assert torch.equal(torch.nan_to_num(got, 0.0), torch.nan_to_num(want, 0.0))


def _layer_like(x, w, H, W, relu):
    """The layer's output in float64 by additions only, a zero coefficient being no operand: x (B, C, H, W), w (16, C, K) -> (B, K, H, W)."""
    nH, nW = (H + 1) // 2, (W + 1) // 2
    d = F.pad(x.double(), (1, 2 * nW - W + 1, 1, 2 * nH - H + 1)).unfold(2, 4, 2).unfold(3, 4, 2)                       # (B, C, nH, nW, 4, 4)
    rows = lambda q: (q[0] - q[2], q[1] + q[2], q[2] - q[1], q[1] - q[3])
    v = [p for r in rows(d.unbind(4)) for p in rows(r.unbind(4))]
    if relu:
        v = [torch.where(p > 0, p, 0.0) for p in v]            # drops NaN, as fmax does
    m = torch.stack([torch.einsum("bchw,ck->bkhw", p, q.double()) for p, q in zip(v, w)]).unflatten(0, (4, 4))
    cols = lambda q: torch.stack((q[0] + q[1] + q[2], q[1] - q[2] - q[3]), -1)
    a = cols(m.unbind(0))                                      # (4, B, K, nH, nW, 2), rows transformed
    return cols(a.unbind(0)).permute(0, 1, 2, 4, 3, 5).reshape(x.shape[0], w.shape[2], 2 * nH, 2 * nW)[:, :, :H, :W]


# the layer on pairs of SMs: rows of each alignment, images copied whole, channels last
PAIR_LAYERS = [((64, 64, 64, 56, 56), "NCHW"), ((130, 44, 72, 14, 14), "NCHW"), ((65, 96, 96, 27, 27), "NCHW"), ((1400, 64, 120, 9, 10), "NCHW"),
               ((513, 64, 128, 11, 12), "NCHW"), ((128, 64, 64, 28, 28), "NHWC"), ((40, 100, 80, 41, 20), "NHWC")]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,layout,kernel", [(*p, "pairs") for p in PAIR_LAYERS] + [((16, 64, 64, 56, 56), "NCHW", "one"), ((48, 16, 16, 48, 48), "NCHW", "one")])
@pytest.mark.parametrize("affine", [False, True])
@pytest.mark.parametrize("relu", [False, True])
def test_image_reaches_the_layer(shape, layout, kernel, affine, relu):
    """NaN and infinities in pixels: without the ReLU NaN comes out as NaN, with it NaN is dropped, and an infinity alone stays one."""
    import wg2x2
    from conftest import kernel_of
    B, C, K, H, W = shape
    assert kernel_of(B, H, W, C, K, layout, affine=affine) == kernel
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    clean, w = rnd(B, C, H, W), rnd(16, C, K) / C ** 0.5
    w[:, :, ::2] = w[:, :, ::2].abs()         # where all terms have one sign an infinity comes out as itself
    si, ti = 1 + 0.2 * rnd(C), 0.3 * rnd(C)
    kw = dict(in_scale=si, in_shift=ti) if affine else {}
    prepared = wg2x2.prepare_weights(w)
    inf = 0x7F800000
    cases = [{(i, 3 + i, 5, 6 - i): n for i, n in enumerate(NANS)},
             {(0, 0, 0, 0): inf, (1, C - 1, H - 1, W - 1): 0xFF800000 - (1 << 32), (2, 7, 4, 3): inf, (3, 8, 3, 4): 0xFF800000 - (1 << 32)},
             {(0, 2, 1, 1): inf, (0, 2, 1, 2): 0xFF800000 - (1 << 32), (1, 5, 3, 3): inf, (1, 5, 4, 3): inf}]             # inf - inf inside a tile
    for case in cases:
        x = clean.clone()
        for at, bits in case.items():
            _put(x, at, bits)
        y = wg2x2.layer_fwd_prepared(x if layout == "NCHW" else x.permute(0, 2, 3, 1).contiguous(), prepared, K, relu=relu, layout=layout, **kw)
        y = (y if layout == "NCHW" else y.permute(0, 3, 1, 2))[:6]
        want = _layer_like(x[:6].double() * si.view(1, -1, 1, 1) + ti.view(1, -1, 1, 1) if affine else x[:6], w, H, W, relu)
        assert not want.isfinite().all() or relu and case is cases[0]
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y[y.isinf()].double(), want[want.isinf()])
        fine = want.isfinite()
        assert float((y[fine] - want[fine]).abs().max()) <= 5e-3 * float(want[fine].abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("shape,layout", PAIR_LAYERS)
def test_padding_stays_zero_under_any_scale(shape, layout):
    """An infinite in_scale (a variance of zero) makes infinities of the channel's pixels, and the padding beside them is still zero."""
    import wg2x2
    B, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, w, si, ti = rnd(B, C, H, W).abs(), rnd(16, C, K).abs() / C, 1 + 0.2 * rnd(C), rnd(C)
    si[5], x[1:, 5], ti[5] = float("inf"), 1.0, 0.0
    x[0, 5] = -1.0
    x[0, 5, 0, 0], x[0, 5, H - 1, W - 1], x[0, 5, 0, W // 2], x[0, 5, H // 2, 0] = 1.0, 1.0, 1.0, 1.0
    y = wg2x2.layer_fwd_prepared(x if layout == "NCHW" else x.permute(0, 2, 3, 1).contiguous(), wg2x2.prepare_weights(w), K, layout=layout, in_scale=si, in_shift=ti)
    y = (y if layout == "NCHW" else y.permute(0, 3, 1, 2))[:3]
    want = _layer_like(x[:3].double() * si.view(1, -1, 1, 1) + ti.view(1, -1, 1, 1), w, H, W, True)
    assert want.isinf().any() and torch.equal(y.isnan(), want.isnan()) and torch.equal(y[y.isinf()].double(), want[want.isinf()])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 49, 196])
def test_relu_mean(n):
    import wg2x2
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((3, 37, n, 1), device="cuda", generator=g)       # 111 planes: 28 warps of four, the last with three
    want = torch.relu(x.double()).mean(dim=(2, 3))
    assert float((wg2x2.relu_mean(x) - want).abs().max()) <= (n + 1) * 2.0 ** -24 * float(x.abs().max())       # n additions and a division
    for i, bits in enumerate(NANS + [0x7F800000, 0xFF800000 - (1 << 32)]):
        bad = x.clone()
        _put(bad, (2, 36 - i, n - 1, 0), bits)
        want = torch.relu(bad).mean(dim=(2, 3))
        got = wg2x2.relu_mean(bad)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
