"""The calls themselves, where several threads make them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
