"""The network's two launch shapes, one group of 13 warps a sample up to one sample per SM and three
groups of five above, at the sizes where they change and where groups end ragged: outputs equal
those of small batches bit for bit (a sample's sums do not depend on its group), gradients the oracle's
to the 1e-2 of test_gpu_cnn, with and without the residual term."""
import numpy as np
import pytest

import cnn_oracle as co
from conftest import gpu_available
from srmg import multigrid as mg
from test_gpu_cnn import batch, rel

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("extra", [-1, 0, 1, 2, 303])
def test_forward_same_in_any_batch(extra):
    net = mg.Cnn(0, seed=7)
    n = sms() + extra
    x, t, xt, tt = batch(n, 5)
    y = net.forward(xt).cpu().numpy()
    for k in (0, n // 2, n - 1):
        yk = net.forward(xt[k:k + 1].contiguous()).cpu().numpy()
        np.testing.assert_array_equal(y[k].view(np.uint32), yk[0].view(np.uint32))


@pytest.mark.parametrize("extra,lam", [(-147, 0.5), (1, 0.0), (1, 0.5)])
def test_gradients_match_oracle(extra, lam):
    import torch
    net = mg.Cnn(0, seed=7)
    theta = net.get_params().astype(np.float64)
    n = max(1, sms() + extra)
    x, t, xt, tt = batch(n, 6)
    ir0 = (np.arange(n, dtype=np.int32) * 16) % 512
    if lam:
        irt = torch.from_numpy(ir0).cuda()
        torch.cuda.synchronize()
        loss, g = net.gradients(xt, tt, lam=lam, ir0=irt, geom=1)
        lo, go = co.gradients(x, t, theta, lam=lam, ir0=ir0, geom=1)
    else:
        loss, g = net.gradients(xt, tt)
        lo, go = co.gradients(x, t, theta)
    assert abs(loss - lo) <= 2e-3 * abs(lo)
    for l, ((w0, w1), (b0, b1)) in enumerate(co.layer_slices()):
        assert rel(g[w0:w1], go[w0:w1]) < 1e-2, (l, "W")
        assert rel(g[b0:b1], go[b0:b1]) < 1e-2, (l, "b")
