"""The weight gradients' sums over samples keep FP32's rounding: a network that passes its output
gradient down every layer unchanged (one unit weight a layer, biases that keep the ReLUs open,
inputs of one), gradients of one sign over many samples, against sums in 64 bits of the bf16
values.

Bars, relative to the sum.  A bias: rounded additions, a chain of 20 pixels and then one value a
sample of the CTA (the smallest share of the 148 CTAs is 11), errors independent of one another:
four standard deviations of sqrt(chain) half units of the last place.  A weight: chains of 5
tensor-core steps a sample over up to 4 samples in the first and last layer and 16 in the others,
each step off by at most one unit, put down by rounded additions."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import multigrid as mg

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

CIN, COUT = (2, 32, 32, 32, 32, 32), (32, 32, 32, 32, 32, 1)
HALF = 2.0 ** -24


@pytest.mark.parametrize("n", [1, 149, 1024, 6000])
def test_sums_over_samples(n):
    import torch
    net = mg.Cnn(0, 1)
    w, b, o = [], [], 0
    for ci, co in zip(CIN, COUT):
        w.append(o + 4 * ci * co)  # centre tap, first output and input channel
        b.append(o + 9 * ci * co)
        o = b[-1] + co
    assert o == net.nparams
    theta = np.zeros(o, np.float32)
    for l in range(6):
        theta[w[l]] = 1.0 if l else 0.0
        theta[b[l]] = (1.0, 0.5, 0.5, 0.5, 0.5, 0.0)[l]
    net.set_params(theta)
    a = (1.0, 1.0, 1.5, 2.0, 2.5, 3.0)  # the layers' inputs
    x = torch.zeros((n, 400, 2), dtype=torch.bfloat16, device="cuda")
    x[:, :, 0] = 1.0
    dy = torch.from_numpy(np.random.default_rng(n).lognormal(0, 2, (n, 16, 16)).astype(np.float32)).cuda()
    net.forward_train(x)
    g = net.backward_step(dy, 0.0, want_grad=True).astype(np.float64)
    total = dy.to(torch.bfloat16).double().sum().item()
    chain = 20 + n / 11 + 1
    for l in range(6):
        assert abs(g[b[l]] / total - 1) <= 4 * HALF * np.sqrt(chain), l
        steps = 5 * min(n, 4 if l in (0, 5) else 16)
        assert abs(g[w[l]] / (a[l] * total) - 1) <= steps * 2 * HALF + 4 * HALF * np.sqrt(chain), l
    net.close()
