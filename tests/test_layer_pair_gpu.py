"""The layer on pairs of SMs (csrc/conv_tc_pair.cuh) through layer_fwd_prepared, at sizes where its cuts can go wrong: row lengths of
each alignment, quads that cross rows and images, images copied whole, channel counts that end inside a slot, a weight stage or a block
of outputs, weights that stay in shared memory and weights that stream, a last unit with one CTA's quads only; both layouts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL_TF32 = 5e-3


# B, C, K, H, W
SHAPES = [
    (96, 64, 64, 40, 56),      # whole 16-byte pieces, weights resident
    (40, 100, 80, 40, 20),     # a slot of four channels at the end, 16 outputs in the last block
    (65, 96, 96, 27, 27),      # odd rows: copies from any 4-byte boundary
    (130, 44, 72, 14, 14),     # rows of 8-byte pieces, quads beyond the image on two sides
    (513, 64, 128, 11, 12),    # nine quads an image: images copied whole
    (1400, 64, 120, 9, 10),
    (1100, 92, 124, 12, 11),   # the same with odd rows, and a slot of four channels
    (17, 256, 256, 28, 31),    # weights stream through their ring
    (24, 64, 64, 65, 64),      # wide rows
]
# channels last: rows of whole quads
CASES = [(s, "NCHW") for s in SHAPES] + [(s, "NHWC") for s in ((96, 64, 64, 40, 56), (40, 100, 80, 41, 20), (513, 64, 128, 11, 12), (17, 256, 256, 27, 32),
                                                               (24, 64, 64, 65, 64), (900, 36, 72, 7, 8), (2000, 64, 68, 5, 4))]


def _inputs(shape, layout="NCHW"):
    import torch
    B, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    return rnd, rnd(B, C, H, W) if layout == "NCHW" else rnd(B, H, W, C), rnd(16, C, K) * (1.0 / (16 * C)) ** 0.5


def _images(B):
    return sorted({0, B // 2, B - 1})      # the oracle computes these


@pytest.mark.parametrize("shape,layout", CASES)
def test_against_the_oracle(oracle, shape, layout):
    import torch
    import wg2x2
    from wg2x2._lib import lib
    B, C, K, H, W = shape
    assert lib.wg2x2_layer_fwd_pair_preferred(B, H, W, C, K, 1 if layout == "NCHW" else 0)
    rnd, x, w = _inputs(shape, layout)
    prepared = wg2x2.prepare_weights(w)
    si, ti, so, to = 1 + 0.2 * rnd(C), 0.3 * rnd(C), 1 + 0.2 * rnd(K), 0.3 * rnd(K)
    r = rnd(B, K, H, W) if layout == "NCHW" else rnd(B, H, W, K)
    pick = _images(B)
    nhwc = lambda t: np.ascontiguousarray((t[pick].permute(0, 2, 3, 1) if layout == "NCHW" else t[pick]).cpu().numpy())
    ch = lambda t: t.view(1, -1, 1, 1) if layout == "NCHW" else t

    def want(a, relu):
        v = oracle.imtrans_fwd(a, relu=relu)
        return oracle.conv_fwd(v, w.cpu().numpy(), H, W)

    for relu in (True, False):
        y = wg2x2.layer_fwd_prepared(x, prepared, K, relu=relu, layout=layout)
        assert wg2x2.last_device_status()[0] == 0
        assert oracle.max_rel(nhwc(y), want(nhwc(x), relu)) <= TOL_TF32
    main = want(nhwc(x * ch(si) + ch(ti)), True) * so.cpu().numpy() + to.cpu().numpy()
    kw = dict(relu=True, layout=layout, in_scale=si, in_shift=ti, out_scale=so, out_shift=to)
    # no shortcut, one of its own, one that Y lies over
    assert oracle.max_rel(nhwc(wg2x2.layer_fwd_prepared(x, prepared, K, **kw)), main) <= TOL_TF32
    for res_relu in (False, True):
        short = torch.relu(r) if res_relu else r
        keep = r.clone()
        y = wg2x2.layer_fwd_prepared(x, prepared, K, residual=r, residual_relu=res_relu, **kw)
        assert oracle.max_rel(nhwc(y), main + nhwc(short)) <= TOL_TF32 and torch.equal(r, keep)
        again = wg2x2.layer_fwd_prepared(x, prepared, K, residual=keep, residual_relu=res_relu, out=keep, **kw)
        # the affine map and the addition, in either order of rounding
        assert again.data_ptr() == keep.data_ptr() and float((again - y).abs().max()) <= 4 * 2.0 ** -24 * float(y.abs().max() + r.abs().max())
    assert torch.equal(wg2x2.layer_fwd_prepared(x, prepared, K, residual=r, residual_relu=True, **kw), y)       # the same bits every time
    assert wg2x2.last_device_status()[0] == 0


@pytest.mark.parametrize("shape,layout", [((96, 64, 64, 40, 56), "NHWC"), ((128, 64, 64, 28, 28), "NHWC"), ((64, 64, 64, 56, 56), "NCHW"), ((65, 96, 96, 27, 27), "NCHW"),
                                          # rows of 8-byte pieces with weights streaming, images copied whole in rows of each alignment
                                          ((128, 256, 256, 14, 14), "NCHW"), ((513, 64, 128, 11, 12), "NCHW"), ((1400, 64, 120, 9, 10), "NCHW"), ((1100, 92, 124, 12, 11), "NCHW")])
def test_every_element_of_many_launches(shape, layout):
    """Against the FP32 kernels: a stage of pixels handed back before its last load has delivered shows in a few pixels of some launches."""
    import torch
    import wg2x2
    B, C, K, H, W = shape
    rnd, x, w = _inputs(shape, layout)
    prepared = wg2x2.prepare_weights(w)
    ch = lambda t: t.view(1, -1, 1, 1) if layout == "NCHW" else t
    si, ti, r = 1 + 0.2 * rnd(C), 0.3 * rnd(C), torch.randn_like(x[:, :1] if layout == "NCHW" else x[..., :1]).expand(*((B, K, H, W) if layout == "NCHW" else (B, H, W, K))).contiguous()
    fp32 = lambda a: wg2x2.conv_fwd(wg2x2.imtrans_fwd(a, relu=True, layout=layout), w, H, W, layout=layout, math="fp32")
    plain, main = fp32(x), fp32(x * ch(si) + ch(ti)) + r
    for _ in range(12):
        for want, kw in ((plain, {}), (main, dict(in_scale=si, in_shift=ti, residual=r))):
            y = wg2x2.layer_fwd_prepared(x, prepared, K, relu=True, layout=layout, **kw)
            assert float((y - want).abs().max()) <= TOL_TF32 * float(want.abs().max())


def _operands64(x, w, H, W, relu, rounded):
    """The layer in float64 sums over the operands that the tensor cores see: weights rounded to TF32, V by FP32 additions and cut to TF32,
    position (1, 1) rounded where `rounded`.  x (B, C, H, W) -> (B, K, H, W)"""
    import torch
    import torch.nn.functional as F
    import wg2x2
    nH, nW = (H + 1) // 2, (W + 1) // 2
    d = F.pad(x, (1, 2 * nW - W + 1, 1, 2 * nH - H + 1)).unfold(2, 4, 2).unfold(3, 4, 2)
    rows = lambda q: (q[0] - q[2], q[1] + q[2], q[2] - q[1], q[1] - q[3])
    v = [p for r in rows(d.unbind(4)) for p in rows(r.unbind(4))]
    if relu:
        v = [p.clamp(min=0) for p in v]
    cut = lambda p: (p.contiguous().view(torch.int32) & -0x2000).view(torch.float32)
    v = [wg2x2.round_tf32(p.contiguous()) if t == 5 and rounded else cut(p) for t, p in enumerate(v)]
    m = torch.stack([torch.einsum("bchw,ck->bkhw", p.double(), wg2x2.round_tf32(q.contiguous()).double()) for p, q in zip(v, w)]).unflatten(0, (4, 4))
    cols = lambda q: torch.stack((q[0] + q[1] + q[2], q[1] - q[2] - q[3]), -1)
    return cols(cols(m.unbind(0)).unbind(0)).permute(0, 1, 2, 4, 3, 5).reshape(x.shape[0], w.shape[2], 2 * nH, 2 * nW)[:, :, :H, :W]


@pytest.mark.parametrize("shape,layout", [((64, 64, 64, 56, 56), "NCHW"), ((130, 44, 72, 14, 14), "NCHW"), ((65, 96, 96, 27, 27), "NCHW"), ((128, 64, 64, 28, 28), "NHWC")])
@pytest.mark.parametrize("relu", [True, False])
def test_operands_are_rounded_as_stated(shape, layout, relu):
    """An accumulator takes 9 C / 8 FP32 additions, each off by a unit in the last place of what it holds at most; that is far less than what
    the rounding of the operands does, and than what cutting position (1, 1) instead would change."""
    import torch
    import wg2x2
    B, C, K, H, W = shape
    rnd, x, w = _inputs(shape, layout)
    y = wg2x2.layer_fwd_prepared(x, wg2x2.prepare_weights(w), K, relu=relu, layout=layout)[:8].double()
    a = x[:8] if layout == "NCHW" else x[:8].permute(0, 3, 1, 2)
    y = y if layout == "NCHW" else y.permute(0, 3, 1, 2)
    want, other = (_operands64(a, w, H, W, relu, rounded) for rounded in (True, False))
    rel = lambda p, q: float((p - q).norm() / q.norm())
    bound = 9 * C / 8 * 2.0 ** -23
    assert rel(other, want) > 4 * bound and rel(y, want) <= bound


def test_output_is_written_exactly():
    """Nothing beyond Y is touched, and all of Y is: plain, with a shortcut in front of the stores or behind them, and with Y over it."""
    import torch
    import wg2x2
    for shape, layout in CASES:
        B, C, K, H, W = shape
        rnd, x, w = _inputs(shape, layout)
        n = B * K * H * W
        room = torch.full((n + 64,), 12345.0, device="cuda")
        y = room[32:32 + n].view((B, K, H, W) if layout == "NCHW" else (B, H, W, K))
        r, prepared, plain = torch.randn_like(y), wg2x2.prepare_weights(w), None
        for residual in (None, r, y):
            y.copy_(r) if residual is y else y.fill_(float("nan"))
            wg2x2.layer_fwd_prepared(x, prepared, K, layout=layout, out=y, residual=residual)
            assert bool(torch.isfinite(y).all()) and bool((room[:32] == 12345.0).all()) and bool((room[32 + n:] == 12345.0).all())
            plain = y.clone() if plain is None else plain
            assert residual is None or torch.equal(y, plain + r)         # one addition, of the same two numbers in either order


@pytest.mark.parametrize("shape,layout", [((96, 64, 64, 40, 56), "NHWC"), ((65, 96, 96, 27, 27), "NCHW"), ((130, 256, 72, 14, 14), "NCHW"), ((64, 64, 64, 56, 56), "NCHW")])
def test_maps_at_any_alignment(shape, layout):
    """out_scale and out_shift off 16 bytes: with the scratch that the query names for the other pointers on 16 bytes (none), the same bits."""
    import ctypes
    import torch
    import wg2x2
    from wg2x2._lib import lib
    B, C, K, H, W = shape
    code, n = 1 if layout == "NCHW" else 0, lambda t: None if t is None else t.data_ptr()
    assert lib.wg2x2_layer_fwd_pair_preferred(B, H, W, C, K, code)
    nv, nw = ctypes.c_size_t(1), ctypes.c_size_t(1)
    lib.wg2x2_layer_fwd_prepared_scratch(B, H, W, C, K, code, 1, ctypes.byref(nv), ctypes.byref(nw))
    assert nv.value == nw.value == 0
    rnd, x, w = _inputs(shape, layout)
    r = rnd(B, K, H, W) if layout == "NCHW" else rnd(B, H, W, K)
    prepared, so, to = wg2x2.prepare_weights(w), 1 + 0.2 * rnd(K), 0.3 * rnd(K)
    off = lambda t: torch.empty(t.numel() + 1, device="cuda")[1:].copy_(t)
    for res in (None, r):
        want = wg2x2.layer_fwd_prepared(x, prepared, K, layout=layout, out_scale=so, out_shift=to, residual=res)
        for s, t in ((off(so), to), (so, off(to)), (off(so), off(to))):
            y = torch.empty_like(want)
            assert lib.wg2x2_layer_fwd_prepared_ex(n(x), None, None, n(prepared), n(y), None, B, H, W, C, K, code, 1, n(s), n(t), n(res), 0, None, 0,
                                                   torch.cuda.current_stream().cuda_stream) == 0
            assert torch.equal(y, want) and torch.equal(wg2x2.layer_fwd_prepared(x, prepared, K, layout=layout, out_scale=s, out_shift=t, residual=res), want)


@pytest.mark.parametrize("shape,layout", [((96, 64, 64, 40, 56), "NHWC"), ((65, 96, 96, 27, 27), "NCHW"), ((130, 72, 72, 14, 14), "NCHW")])
def test_output_over_the_input_needs_scratch(shape, layout):
    """Layers that only transform and products in memory could compute over their own input: refused without V_scratch, X left as it is."""
    import torch
    import wg2x2
    from wg2x2._lib import lib
    B, C, K, H, W = shape
    assert lib.wg2x2_layer_fwd_pair_preferred(B, H, W, C, K, 1 if layout == "NCHW" else 0)
    rnd, x, w = _inputs(shape, layout)
    prepared, y, n = wg2x2.prepare_weights(w), x.clone(), lambda t: None if t is None else t.data_ptr()
    call = lambda v: lib.wg2x2_layer_fwd_prepared_ex(n(y), None, None, n(prepared), n(y), n(v), B, H, W, C, K, 1 if layout == "NCHW" else 0, 1,
                                                     None, None, None, 0, None, 0, torch.cuda.current_stream().cuda_stream)
    assert call(None) == -2
    torch.cuda.synchronize()
    assert torch.equal(x, y)
    assert call(torch.empty((16, B, (H + 1) // 2, (W + 1) // 2, C), device="cuda")) == 0
    want = wg2x2.layer_fwd_prepared(x, prepared, K, layout=layout)
    assert float((y - want).abs().max()) <= TOL_TF32 * float(want.abs().max())


@pytest.mark.parametrize("shape,layout", [((111, 128, 128, 10, 10), "NCHW"), ((48, 256, 256, 14, 14), "NCHW"), ((128, 256, 256, 14, 14), "NCHW"), ((46, 96, 192, 12, 12), "NHWC")])
def test_rule_sees_the_options(shape, layout):
    """Plain layers that run on pairs of SMs, and with a map or a shortcut on the path that is then the faster: what the queries say fits together,
    and either kernel's results agree."""
    import ctypes
    import torch
    import wg2x2
    from wg2x2._lib import lib
    B, C, K, H, W = shape
    sizes = (B, H, W, C, K, 1 if layout == "NCHW" else 0)
    for_ = {(a, s): lib.wg2x2_layer_fwd_pair_preferred_for(*sizes, a, s) for a in (0, 1) for s in (0, 1, 2)}
    every = int(all(for_.values()))
    assert lib.wg2x2_layer_fwd_pair_preferred(*sizes) == lib.wg2x2_layer_fwd_pair_preferred_for(*sizes, 0, -1) == every
    assert for_[0, 0] == (layout == "NCHW") and every == (shape == (128, 256, 256, 14, 14))
    nv, nw = ctypes.c_size_t(), ctypes.c_size_t()
    lib.wg2x2_layer_fwd_prepared_scratch(*sizes, 1, ctypes.byref(nv), ctypes.byref(nw))
    assert (nv.value == 0) == bool(every)         # what the query names is enough for any options
    rnd, x, w = _inputs(shape, layout)
    prepared, r = wg2x2.prepare_weights(w), rnd(B, K, H, W) if layout == "NCHW" else rnd(B, H, W, K)
    plain = wg2x2.layer_fwd_prepared(x, prepared, K, layout=layout)
    kw = dict(layout=layout, residual=r, in_scale=torch.ones(C, device="cuda"), in_shift=torch.zeros(C, device="cuda"))
    tol = 2e-3 * float(plain.abs().max())          # another kernel: one rounds where the other cuts
    assert float((wg2x2.layer_fwd_prepared(x, prepared, K, **kw) - (plain + r)).abs().max()) <= tol
    got = wg2x2.layer_fwd_prepared(x, prepared, K, out=r, **dict(kw, residual=r))
    assert got.data_ptr() == r.data_ptr() and bool(torch.isfinite(got).all())


def test_zero_blocks_are_skipped_right(oracle):
    import wg2x2
    shape = (64, 160, 128, 28, 28)
    B, C, K, H, W = shape
    rnd, x, w = _inputs(shape)
    for t in range(16):          # every block of 64 outputs x 32 inputs but a few; all of position 5
        for kb in range(2):
            for cc in range(5):
                if t == 5 or (t + kb + cc) % 3:
                    w[t, 32 * cc:32 * cc + 32, 64 * kb:64 * kb + 64] = 0
    y = wg2x2.layer_fwd_prepared(x, wg2x2.prepare_weights(w), K, layout="NCHW")
    nhwc = lambda t: np.ascontiguousarray(t[_images(B)].permute(0, 2, 3, 1).cpu().numpy())
    assert oracle.max_rel(nhwc(y), oracle.conv_fwd(oracle.imtrans_fwd(nhwc(x), relu=True), w.cpu().numpy(), H, W)) <= TOL_TF32


@pytest.mark.parametrize("shape,nth", [(SHAPES[0], 0), (SHAPES[0], 3), (SHAPES[7], 0), (SHAPES[7], 10)])        # weights resident, weights streaming
def test_times_out_and_recovers(shape, nth):
    """CTA 0's weight producer stops before one load, with nothing in flight, under a limit of a few thousand polls."""
    import torch
    import wg2x2
    from wg2x2._lib import lib
    rnd, x, w = _inputs(shape)
    prepared, K = wg2x2.prepare_weights(w), shape[2]
    want = wg2x2.layer_fwd_prepared(x, prepared, K, layout="NCHW")
    torch.cuda.synchronize()
    try:
        lib.wg2x2_set_wait_limit(20000)
        lib.wg2x2_test_drop_load(nth)
        wg2x2.layer_fwd_prepared(x, prepared, K, layout="NCHW")
        st, where = wg2x2.last_device_status()
        assert st == -4
        # whichever role ran out first: an issuer (0x10 .. 0x13), a transform team (0x0B, 0x0C), a producer (0x09, 0x0A) or the epilogue (0x04)
        assert (where >> 8) in (0x10, 0x11, 0x12, 0x13, 0x0C, 0x0B, 0x0A, 0x09, 0x04), "0x%x" % where
    finally:
        lib.wg2x2_test_drop_load(-1)
        lib.wg2x2_set_wait_limit(0)
    assert torch.equal(wg2x2.layer_fwd_prepared(x, prepared, K, layout="NCHW"), want) and wg2x2.last_device_status()[0] == 0
