"""A training step on more samples than the backward pass takes at a time: the gradient is the sum
of the parts' gradients, and the scratch memory stays below 205 KB a sample (the activations of
six layers and the gradients of two)."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import multigrid as mg

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def test_parts_add_up():
    import torch
    n, at = 20_000, (0, 8192, 16384, 20_000)
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((n, 400, 2), generator=gen, device="cuda").to(torch.bfloat16)
    dy = torch.randn((n, 16, 16), generator=gen, device="cuda")
    torch.cuda.empty_cache()
    net = mg.Cnn(0, 7)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    net.forward_train(x)
    used = free - torch.cuda.mem_get_info()[0]
    whole = net.backward_step(dy, 0.0, want_grad=True).astype(np.float64)
    assert used < n * (8 * 25_600 + 5_000)
    parts = np.zeros_like(whole)
    for lo, hi in zip(at, at[1:]):
        net.forward_train(x[lo:hi].contiguous())
        parts += net.backward_step(dy[lo:hi].contiguous(), 0.0, want_grad=True)
    # the same partial sums, added in FP32 by one side: two roundings
    assert np.abs(whole - parts).max() <= 2 * 2.0 ** -24 * np.abs(parts).max()
    net.close()
