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
