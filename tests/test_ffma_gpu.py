"""The FP32 kernels of the Winograd-domain product at the edges of their tiles: every block height (64, 32 and 16 rows, picked
from the number of results), rows, columns and contractions that end inside a tile or a stage, odd images, and channel
counts that are no multiple of four (which leave TMA for plain copies), against the float64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5
# (B, H, W, C, K): block heights of the forward product (rows = tiles) as commented
SHAPES = [
    (8, 55, 56, 20, 30),       # 64 rows, neither channel count fits a tile; K not a multiple of 4
    (8, 55, 56, 36, 32),       # 64 rows, TMA
    (4, 55, 56, 17, 31),       # 32 rows, plain copies
    (4, 56, 56, 16, 40),       # 32 rows, one stage of 16 steps exactly
    (1, 5, 7, 40, 68),         # 16 rows, a single ragged block
    (2, 9, 9, 13, 5),          # 16 rows, plain copies, fewer columns than a block
    (1, 1, 1, 4, 4),           # one tile
]


@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
@pytest.mark.parametrize("shape", SHAPES)
def test_products_at_tile_edges(oracle, shape, layout):
    import torch
    import wg2x2
    B, H, W, C, K = shape
    rng = np.random.default_rng(sum(shape))
    X = rng.standard_normal((B, H, W, C)).astype(np.float32)
    Wt = (0.1 * rng.standard_normal((16, C, K))).astype(np.float32)
    mask = (rng.random((16, C, K)) < 0.5).astype(np.float32)
    dY = rng.standard_normal((B, H, W, K)).astype(np.float32)
    V = oracle.imtrans_fwd(X, relu=True, dtype=np.float32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    img = lambda a: dev(a if layout == "NHWC" else np.transpose(a, (0, 3, 1, 2)))
    Y = wg2x2.conv_fwd(dev(V), dev(Wt), H, W, layout=layout, math="fp32").cpu().numpy()
    Y = Y if layout == "NHWC" else np.transpose(Y, (0, 2, 3, 1))
    assert oracle.max_rel(Y, oracle.conv_fwd(V, Wt, H, W)) <= TOL
    dVo, dWo = oracle.conv_bwd(V, Wt, dY, mask=mask)
    dV, dW = wg2x2.conv_bwd(dev(V), dev(Wt), img(dY), mask=dev(mask), layout=layout, relu=True, math="fp32")
    assert oracle.max_rel(dW.cpu().numpy(), dWo) <= TOL
    assert oracle.max_rel(dV.cpu().numpy(), np.where(V > 0, dVo, 0)) <= TOL
    assert wg2x2.last_device_status()[0] == 0
