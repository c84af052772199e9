"""The NCHW kernels that walk tiles with lane = channel, at sizes so small that a tile row is cut into segments (one image,
few channels), and at widths that leave a ragged last segment, against the float64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 9, 41, 32), (1, 64, 64, 16), (2, 3, 100, 36), (1, 7, 150, 68), (3, 27, 27, 32), (1, 1, 35, 4)])
def test_segmented_rows(oracle, shape):
    import torch
    import wg2x2
    B, H, W, C = shape
    rng = np.random.default_rng(sum(shape))
    nH, nW = (H + 1) // 2, (W + 1) // 2
    dV = rng.standard_normal((16, B, nH, nW, C)).astype(np.float32)
    V = rng.standard_normal((16, B, nH, nW, C)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    for mask in (None, V):
        dX = wg2x2.imtrans_bwd(dev(dV), H, W, V_relu=None if mask is None else dev(mask), layout="NCHW").cpu().numpy()
        assert oracle.max_rel(np.transpose(dX, (0, 2, 3, 1)), oracle.imtrans_bwd(dV, H, W, Vmask=mask)) <= 1e-5
    # dM, through the tensor-core gradients
    Wt = (0.1 * rng.standard_normal((16, C, C))).astype(np.float32)
    dY = rng.standard_normal((B, H, W, C)).astype(np.float32)
    dVo, dWo = oracle.conv_bwd(V, Wt, dY)
    gV, gW = wg2x2.conv_bwd(dev(V), dev(Wt), dev(np.transpose(dY, (0, 3, 1, 2))), layout="NCHW", math="tf32")
    assert oracle.max_rel(gV.cpu().numpy(), dVo) <= 5e-3
    assert oracle.max_rel(gW.cpu().numpy(), dWo) <= 5e-3
    assert wg2x2.last_device_status()[0] == 0


# few tiles: the wide path with 64, 128 and 256 columns per unit, channel counts that end inside a tile, a chunk and a byte of
# the zero-block map (the last shape has more than 64 chunks: no map); every third 64 x 32 weight block is empty
@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 4, 4), (3, 11, 11, 512, 96), (1, 14, 14, 300, 68), (2, 27, 26, 128, 132), (4, 14, 15, 64, 516),
                                   (16, 7, 7, 260, 260), (1, 8, 8, 36, 4), (1, 3, 3, 2080, 64)])
def test_few_tiles(oracle, shape, layout):
    import torch
    import wg2x2
    B, H, W, C, K = shape
    rng = np.random.default_rng(sum(shape))
    X = rng.standard_normal((B, H, W, C)).astype(np.float32)
    Wt = (rng.standard_normal((16, C, K)) / np.sqrt(C)).astype(np.float32)
    for t in range(16):
        for cc in range(0, C, 32):
            for kb in range(0, K, 64):
                if (t + cc // 32 + kb // 64) % 3 == 0:
                    Wt[t, cc:cc + 32, kb:kb + 64] = 0
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    img = lambda a: dev(a if layout == "NHWC" else np.transpose(a, (0, 3, 1, 2)))
    back = lambda t: t.cpu().numpy() if layout == "NHWC" else np.transpose(t.cpu().numpy(), (0, 2, 3, 1))
    V = oracle.imtrans_fwd(X, relu=True, dtype=np.float32)
    want = oracle.conv_fwd(V, Wt, H, W)
    assert wg2x2._lib.lib.wg2x2_conv_fwd_prepared_workspace_bytes(B, (H + 1) // 2, (W + 1) // 2, C, K) > 0
    prepared = wg2x2.prepare_weights(dev(Wt))
    for Y in (wg2x2.conv_fwd(dev(V), dev(Wt), H, W, layout=layout, math="tf32"),
              wg2x2.conv_fwd_prepared(dev(V), prepared, K, H, W, layout=layout),
              wg2x2.conv_fwd_prepared(dev(V), prepared, K, H, W, layout=layout, wide=False),
              wg2x2.layer_fwd_prepared(img(X), prepared, K, relu=True, layout=layout)):
        assert oracle.max_rel(back(Y), want) <= 5e-3
    assert wg2x2.last_device_status()[0] == 0


# the pruning mask folded into the product op against W * mask as torch's autograd has it
@pytest.mark.parametrize("math", ["fp32", "tf32"])
@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("C,K", [(4, 4), (36, 20), (96, 72)])
def test_masked_layer(C, K, layout, math):
    import torch
    import wg2x2
    from winograd_conv import WinogradConvLayer
    g = torch.Generator(device="cuda").manual_seed(C + K)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    V, W = rnd(16, 2, 4, 5, C).requires_grad_(True), rnd(16, C, K)
    mask = (torch.rand((16, C, K), generator=g, device="cuda") < 0.4).float()
    dY = rnd(2, 7, 10, K) if layout == "NHWC" else rnd(2, K, 7, 10)
    layer = WinogradConvLayer(C, K, mask=mask, W_init=lambda s: W, device="cuda")
    y = layer(V, out_hw=(7, 10), data_format=layout, math=math)
    y2 = wg2x2.ops.conv_op(V, layer.W * layer.mask, 7, 10, layout, math)
    assert torch.equal(y, y2)
    for a, b in zip(torch.autograd.grad(y, (V, layer.W), dY), torch.autograd.grad(y2, (V, layer.W), dY)):
        assert torch.equal(a, b)


# the ReLU mask as bits, forward and gradient, through every kernel that writes or reads them: vector and scalar channels, rows cut
# into segments, bands, walks along a row with one and two channels per lane, whole small images, rows wider than a band
@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("shape", [(2, 9, 13, 32), (3, 6, 7, 5), (1, 64, 64, 16), (2, 28, 28, 36), (32, 28, 30, 32), (40, 21, 27, 64), (75, 14, 14, 256),
                                   (300, 7, 7, 33), (1, 3, 200, 8), (20, 45, 44, 68)])
def test_relu_bits(oracle, shape, layout):
    import torch
    import wg2x2
    B, H, W, C = shape
    rng = np.random.default_rng(sum(shape))
    X = rng.standard_normal((B, H, W, C)).astype(np.float32)
    G = rng.standard_normal((16, B, (H + 1) // 2, (W + 1) // 2, C)).astype(np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    img = lambda a: dev(a if layout == "NHWC" else np.transpose(a, (0, 3, 1, 2)))
    back = lambda t: t.cpu().numpy() if layout == "NHWC" else np.transpose(t.cpu().numpy(), (0, 2, 3, 1))
    for relu in (True, False):
        x = img(X).requires_grad_(True)
        v = wg2x2.ops.imtrans_op(x, relu, layout)
        assert torch.equal(v, wg2x2.imtrans_fwd(x.detach(), relu=relu, layout=layout))
        V = v.detach().cpu().numpy()
        dx, = torch.autograd.grad(v, x, dev(G))
        assert oracle.max_rel(back(dx), oracle.imtrans_bwd(G, H, W, Vmask=V if relu else None)) <= 1e-5
