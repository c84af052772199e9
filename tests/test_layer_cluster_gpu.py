"""The one-kernel layer for few tiles (clusters of four CTAs) through layer_fwd_prepared, at sizes where its cuts can go wrong: every
cut of tiles x channels, tiles and channels that end inside one, odd images, one chunk of input channels and more than its
operand stages hold, plain and with every option, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 4, 1), (2, 9, 13, 32, 36), (1, 14, 14, 256, 256), (5, 27, 27, 48, 80), (1, 56, 56, 64, 64),
                                   (4, 40, 38, 64, 64), (3, 33, 64, 20, 100), (2, 8, 9, 448, 64), (16, 23, 23, 48, 32), (7, 7, 7, 128, 130)])
def test_layer_of_few_tiles(oracle, shape, layout):
    import torch
    import wg2x2
    B, H, W, C, K = shape
    rng = np.random.default_rng(sum(shape))
    X = rng.standard_normal((B, H, W, C)).astype(np.float32)
    Wt = (rng.standard_normal((16, C, K)) / np.sqrt(C)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    img = lambda a: dev(a if layout == "NHWC" else np.transpose(a, (0, 3, 1, 2)))
    back = lambda t: t.cpu().numpy() if layout == "NHWC" else np.transpose(t.cpu().numpy(), (0, 2, 3, 1))
    prepared = wg2x2.prepare_weights(dev(Wt))
    for relu in (True, False):
        Y = wg2x2.layer_fwd_prepared(img(X), prepared, K, relu=relu, layout=layout)
        assert oracle.max_rel(back(Y), oracle.conv_fwd(oracle.imtrans_fwd(X, relu=relu), Wt, H, W)) <= 5e-3
    si, ti = (1 + 0.3 * rng.standard_normal(C)).astype(np.float32), (0.5 * rng.standard_normal(C)).astype(np.float32)
    so, to = (1 + 0.2 * rng.standard_normal(K)).astype(np.float32), (0.3 * rng.standard_normal(K)).astype(np.float32)
    R = rng.standard_normal((B, H, W, K)).astype(np.float32)
    want = oracle.conv_fwd(oracle.imtrans_fwd(X * si + ti, relu=True), Wt, H, W) * so + to
    for res_relu in (False, True):
        Y = wg2x2.layer_fwd_prepared(img(X), prepared, K, relu=True, layout=layout, in_scale=dev(si), in_shift=dev(ti), out_scale=dev(so),
                                     out_shift=dev(to), residual=img(R), residual_relu=res_relu)
        assert oracle.max_rel(back(Y), want + (np.maximum(R, 0) if res_relu else R)) <= 5e-3
    assert wg2x2.last_device_status()[0] == 0


# residual_relu where the other paths run: one-kernel NCHW layer, wide path, transform + row-walk kernel, pairs of SMs
@pytest.mark.parametrize("shape,layout,kernel", [((16, 56, 56, 64, 64), "NCHW", "one"), ((24, 14, 14, 256, 256), "NCHW", "wide"), ((48, 14, 14, 256, 256), "NHWC", "wide"),
                                                 ((24, 48, 46, 64, 64), "NHWC", "walk"), ((40, 49, 49, 32, 64), "NCHW", "walk"), ((40, 13, 15, 256, 256), "NCHW", "wide"),
                                                 ((48, 14, 14, 256, 256), "NCHW", "pairs"), ((24, 48, 48, 64, 64), "NHWC", "pairs")])
def test_residual_relu_of_the_other_paths(shape, layout, kernel):
    import torch
    import wg2x2
    from conftest import kernel_of
    assert kernel_of(*shape, layout, shortcut=1) == kernel
    B, H, W, C, K = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, r = (rnd(B, H, W, c) if layout == "NHWC" else rnd(B, c, H, W) for c in (C, K))
    prepared = wg2x2.prepare_weights(rnd(16, C, K) / C ** 0.5)
    sc, sh = 1 + 0.2 * rnd(K), 0.3 * rnd(K)
    kw = dict(relu=True, layout=layout, out_scale=sc, out_shift=sh)
    got = wg2x2.layer_fwd_prepared(x, prepared, K, residual=r, residual_relu=True, **kw)
    assert torch.equal(got, wg2x2.layer_fwd_prepared(x, prepared, K, residual=torch.relu(r), **kw))


# the output transform of the wide path, NCHW against NHWC (the same sums in the same order), odd sizes and one band or several
@pytest.mark.parametrize("shape", [(64, 13, 15, 256, 256), (40, 27, 26, 256, 320), (500, 7, 7, 256, 256), (9, 57, 56, 256, 256)])
def test_output_transform_layouts_agree(shape):
    import torch
    import wg2x2
    B, H, W, C, K = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    v, prepared = rnd(16, B, (H + 1) // 2, (W + 1) // 2, C), wg2x2.prepare_weights(rnd(16, C, K) / C ** 0.5)
    sc, sh, r = 1 + 0.2 * rnd(K), 0.3 * rnd(K), rnd(B, H, W, K)
    for kw in ({}, dict(out_scale=sc, out_shift=sh, residual=r)):
        a = wg2x2.conv_fwd_prepared(v, prepared, K, H, W, layout="NHWC", **kw)
        if kw:
            kw["residual"] = r.permute(0, 3, 1, 2).contiguous()
        b = wg2x2.conv_fwd_prepared(v, prepared, K, H, W, layout="NCHW", **kw)
        assert torch.equal(a.permute(0, 3, 1, 2), b)
