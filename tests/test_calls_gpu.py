"""The calls themselves: made by several threads, with operands off 16-byte boundaries, and what autograd and its tools ask of them."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t):
    """The same values one float off a 16-byte boundary."""
    o = torch.empty(t.numel() + 1, device=t.device)[1:].view(t.shape)
    assert o.data_ptr() % 16 == 4
    return o.copy_(t)


def _on_new_thread():
    """A thread that runs one function after another: call(f) returns f()."""
    from concurrent.futures import ThreadPoolExecutor
    pool = ThreadPoolExecutor(1)
    return lambda f: pool.submit(f).result()


def test_two_threads_with_different_sizes_of_one_kernel():
    """The 1x1 kernel takes 24 KB of shared memory per 32 channels: 193 KB in one thread, then 97 KB in another, then 193 KB again."""
    import wg2x2
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((1, 256, 7, 7), device="cuda", generator=g)
    w = wg2x2.round_tf32(torch.randn((64, 256, 1, 1), device="cuda", generator=g))
    big, small = lambda: wg2x2.conv1x1(x, w), lambda: wg2x2.conv1x1(x[:, :128].contiguous(), w[:, :128].contiguous())
    a, b = _on_new_thread(), _on_new_thread()
    first = a(big)
    b(small)
    assert torch.equal(a(big), first) and torch.equal(b(big), first)


# few tiles (clusters), many (the one kernel), many channels (wide path), a layout the one kernel does not take
@pytest.mark.parametrize("shape,layout,one_kernel", [((1, 64, 64, 56, 56), "NCHW", False), ((64, 64, 64, 56, 56), "NCHW", True),
                                                     ((128, 256, 256, 14, 14), "NCHW", False), ((64, 64, 64, 56, 56), "NHWC", False)])
def test_fused_preferred(shape, layout, one_kernel):
    import wg2x2
    B, C, K, H, W = shape
    assert wg2x2.fused_preferred(B, H, W, C, K, layout) == one_kernel


# NCHW layers whose rows are whole 16-byte pieces have read out_scale, out_shift and residual at any alignment since the one-kernel layer
# was their only path; the sizes here are now computed on clusters, by the wide path and by the one kernel
@pytest.mark.parametrize("shape", [(48, 512, 128, 16, 16), (3, 512, 64, 28, 28), (1, 64, 64, 56, 56), (5, 48, 80, 28, 28), (16, 64, 64, 56, 56), (2, 128, 320, 8, 8)])
def test_extras_at_any_alignment(shape):
    import wg2x2
    B, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, r, prepared = rnd(B, C, H, W), rnd(B, K, H, W), wg2x2.prepare_weights(rnd(16, C, K) / C ** 0.5)
    sc, sh, isc, ish = 1 + 0.2 * rnd(K), 0.3 * rnd(K), 1 + 0.2 * rnd(C), 0.3 * rnd(C)
    kw = dict(relu=True, layout="NCHW", in_scale=isc, in_shift=ish)
    for relu in (False, True):
        want = wg2x2.layer_fwd_prepared(x, prepared, K, out_scale=sc, out_shift=sh, residual=r, residual_relu=relu, **kw)
        scale = float(want.abs().max())
        for s, t, q in ((_off(sc), sh, r), (sc, _off(sh), r), (sc, sh, _off(r)), (_off(sc), _off(sh), _off(r))):
            got = wg2x2.layer_fwd_prepared(x, prepared, K, out_scale=s, out_shift=t, residual=q, residual_relu=relu, **kw)
            # another path at worst: V rounded to 11 bits where the other cuts it, 2^-11 of each of C x 16 terms of random sign
            assert float((got - want).abs().max()) <= 2e-3 * scale
        got = wg2x2.layer_fwd_prepared(x, prepared, K, out_scale=sc, out_shift=sh, residual=r, residual_relu=relu, relu=True, layout="NCHW",
                                       in_scale=_off(isc), in_shift=_off(ish))
        assert float((got - want).abs().max()) <= 2e-3 * scale


# few tiles, the one kernel's sizes, many channels: where the layer could run as one kernel, a CTA would read pixels that another has written over
@pytest.mark.parametrize("layout", ["NCHW", "NHWC"])
@pytest.mark.parametrize("shape", [(2, 32, 9, 13), (1, 64, 56, 56), (16, 64, 56, 56), (4, 256, 14, 14), (2, 256, 8, 8)])
def test_output_over_the_input(shape, layout):
    import wg2x2
    B, C, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, prepared = rnd(B, C, H, W) if layout == "NCHW" else rnd(B, H, W, C), wg2x2.prepare_weights(rnd(16, C, C) / C ** 0.5)
    for residual in (None, x.clone()):
        want = wg2x2.layer_fwd_prepared(x, prepared, C, layout=layout, residual=residual)
        y = x.clone()
        got = wg2x2.layer_fwd_prepared(y, prepared, C, layout=layout, out=y, residual=None if residual is None else y)
        assert got.data_ptr() == y.data_ptr()
        assert float((got - want).abs().max()) <= 2e-3 * float(want.abs().max())        # another path at worst, as above


def test_extras_off_16_bytes_stay_refused_where_only_the_wide_path_runs():
    import wg2x2
    x, prepared = torch.zeros((48, 256, 16, 16), device="cuda"), wg2x2.prepare_weights(torch.zeros((16, 256, 256), device="cuda"))
    s = torch.ones(256, device="cuda")
    with pytest.raises(wg2x2.Wg2x2Error) as e:
        wg2x2.layer_fwd_prepared(x, prepared, 256, layout="NCHW", out_scale=_off(s), out_shift=s)
    assert e.value.status == -1


@pytest.mark.parametrize("layout", ["NCHW", "NHWC"])
@pytest.mark.parametrize("shape", [(1, 64, 64, 56, 56), (2, 32, 96, 9, 13), (16, 64, 64, 56, 56), (24, 256, 256, 14, 14), (24, 64, 64, 28, 28)])
def test_residual_block(shape, layout):
    """Both layers one by one, with the ReLUs and the addition by torch: the same kernels where the shortcut is a tensor (written in place),
    and relu(x) where there is none."""
    import wg2x2
    B, C, K, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    img = lambda c: rnd(B, c, H, W) if layout == "NCHW" else rnd(B, H, W, c)
    x, short = img(C), img(K)
    pa, pb = wg2x2.prepare_weights(rnd(16, C, K) / C ** 0.5), wg2x2.prepare_weights(rnd(16, K, K) / K ** 0.5)
    bn = lambda c: (1 + 0.2 * rnd(c), 0.3 * rnd(c))
    a, b, o = bn(C), bn(K), bn(K)
    mid = wg2x2.layer_fwd_prepared(x, pa, K, relu=True, layout=layout, in_scale=a[0], in_shift=a[1])
    main = wg2x2.layer_fwd_prepared(mid, pb, K, relu=True, layout=layout, in_scale=b[0], in_shift=b[1], out_scale=o[0], out_shift=o[1])
    tol = 4 * 2.0 ** -24 * float(main.abs().max() + short.abs().max() + x.abs().max())         # the affine map and the addition, rounded once or twice
    keep, x0 = short.clone(), x.clone()
    y = wg2x2.residual_block(x, short, pa, a, pb, b, o, K, layout=layout)
    assert y.data_ptr() == short.data_ptr() and torch.equal(x, x0)
    assert float((y - (main + keep)).abs().max()) <= tol
    if C == K:
        y = wg2x2.residual_block(x, None, pa, a, pb, b, o, K, layout=layout)
        assert y.data_ptr() != x.data_ptr() and torch.equal(x, x0)
        assert float((y - (main + torch.relu(x))).abs().max()) <= tol
    else:
        with pytest.raises(ValueError):
            wg2x2.residual_block(x, None, pa, a, pb, b, o, K, layout=layout)


def _layer(g, C=16, K=8):
    import winograd_conv
    import winograd_imtrans
    layer = winograd_conv.WinogradConvLayer(C, K, device="cuda", W_init=lambda s: torch.randn(s, generator=g, device="cuda"))
    return layer, lambda x: layer(winograd_imtrans.WinogradImTrans(x, nl=torch.relu, data_format="NHWC"), out_hw=x.shape[1:3])


def test_backward_of_one_graph_on_several_threads():
    """Each thread has the gradients, or is told that the graph is gone."""
    g = torch.Generator(device="cuda").manual_seed(5)
    layer, f = _layer(g)
    x = torch.randn((3, 9, 8, 16), generator=g, device="cuda", requires_grad=True)
    y = f(x)
    dy = torch.randn(y.shape, generator=g, device="cuda")
    want = torch.autograd.grad(y, (x, layer.W), dy, retain_graph=True)
    bad = []

    def run(retain, lost_is_fine, y):
        try:
            got = torch.autograd.grad(y, (x, layer.W), dy, retain_graph=retain)
            if not all(torch.equal(p, q) for p, q in zip(got, want)):
                bad.append("other values")
        except RuntimeError as e:
            if not lost_is_fine or "second time" not in str(e):
                bad.append(e)

    for retain in (True, False):
        for _ in range(20):
            yy = y if retain else f(x)
            ts = [threading.Thread(target=run, args=(retain, not retain, yy)) for _ in range(4)]
            [t.start() for t in ts]
            [t.join() for t in ts]
    assert not bad, bad[0]


def test_saved_tensor_hooks_see_everything_that_is_saved():
    """The transform's ReLU mask, and the product's two operands, pass through the hooks (offloading, checkpointing) in both directions."""
    g = torch.Generator(device="cuda").manual_seed(6)
    layer, f = _layer(g)
    x = torch.randn((3, 9, 8, 16), generator=g, device="cuda", requires_grad=True)
    y = f(x)
    dy = torch.randn(y.shape, generator=g, device="cuda")
    want = torch.autograd.grad(y, (x, layer.W), dy)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
        y = f(x)
    assert len(packed) == 3
    assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(y, (x, layer.W), dy), want))


def test_forward_mode_is_refused():
    import torch.autograd.forward_ad as fw
    import wg2x2
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, v, w, m = rnd(2, 8, 8, 16), rnd(16, 2, 4, 4, 16), rnd(16, 16, 8), torch.ones((16, 16, 8), device="cuda")
    with fw.dual_level():
        dual = lambda t: fw.make_dual(t, torch.ones_like(t))
        for call in (lambda: wg2x2.ops.imtrans_op(dual(x), True), lambda: wg2x2.ops.conv_op(dual(v), w), lambda: wg2x2.ops.conv_op(v, dual(w)),
                     lambda: wg2x2.ops.conv_op(v, w, mask=dual(m))):
            with pytest.raises(NotImplementedError):
                call()
        wg2x2.ops.conv_op(wg2x2.ops.imtrans_op(x, True), w, mask=m)


@pytest.mark.parametrize("layout,masked", [("NHWC", False), ("NHWC", True), ("NCHW", True)])
def test_traced_module(layout, masked):
    """torch.jit.trace records both ops: other inputs give other outputs and gradients, with gradients off too."""
    import winograd_conv
    import winograd_imtrans
    g = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.layer = winograd_conv.WinogradConvLayer(16, 8, device="cuda", W_init=lambda s: rnd(*s), mask=(rnd(16, 16, 8) > 0).float() if masked else None)

        def forward(self, x):
            v = winograd_imtrans.WinogradImTrans(2 * x, nl=torch.relu, data_format=layout)
            return torch.tanh(self.layer(v, out_hw=x.shape[1:3] if layout == "NHWC" else x.shape[2:], data_format=layout))

    net, shape = Net(), (2, 9, 8, 16) if layout == "NHWC" else (2, 16, 9, 8)
    for grad in (True, False):
        with torch.set_grad_enabled(grad):
            traced = torch.jit.trace(net, (rnd(*shape),))
        x = rnd(*shape).requires_grad_(True)
        y, z = net(x), traced(x)
        assert torch.equal(y, z)
        if grad:
            dy = torch.randn_like(y)
            want = torch.autograd.grad(y, (x, net.layer.W), dy)
            assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(z, (x, net.layer.W), dy), want))
