import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sparse-winograd-cnn_b200")
for p in (ROOT, PKG):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def oracle():
    from oracle import wg_oracle
    wg_oracle.lib()
    return wg_oracle


def kernel_of(B, H, W, C, K, layout, affine=0, shortcut=0):
    """Which way layer_fwd_prepared takes an aligned layer with these options: "pairs", "clusters" or "one" (kernel), or through memory "wide" or "walk"."""
    import ctypes
    from wg2x2._lib import lib
    code = 1 if layout == "NCHW" else 0
    if lib.wg2x2_layer_fwd_pair_preferred_for(B, H, W, C, K, code, affine, shortcut):
        return "pairs"
    v, ws = ctypes.c_size_t(), ctypes.c_size_t()
    lib.wg2x2_layer_fwd_prepared_scratch(B, H, W, C, K, code, 1, ctypes.byref(v), ctypes.byref(ws))
    if not v.value:
        return "one" if lib.wg2x2_layer_fwd_fused_preferred(B, H, W, C, K, code) else "clusters"
    return "wide" if ws.value else "walk"


def pytest_collection_modifyitems(config, items):
    # keep the file order alphabetical so that test_zz_* files run last
    items.sort(key=lambda it: (os.path.basename(str(it.fspath)),))
