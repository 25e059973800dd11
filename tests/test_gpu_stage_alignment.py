"""The stage kernels' wide copies (16 bytes where every field allows them, else 8): fields that start
at an odd double give the results of aligned ones bit for bit, and flux gives the same fluxes
and minimum with and without the per-block time steps."""
import ctypes

import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg.streamer import MINIMAL

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def shifted(a, by):
    """A copy of a on the device, by doubles after a 16-byte boundary."""
    import torch
    flat = torch.zeros(a.size + 2, dtype=torch.float64, device="cuda")
    t = flat[by:by + a.size].view(*a.shape)
    t.copy_(torch.from_numpy(a))
    assert t.data_ptr() % 16 == 8 * by
    return t


@pytest.mark.parametrize("kernel", ["netcharge", "electric_field", "flux", "rates"])
def test_odd_start_bit_identical(kernel):
    import torch
    p = gen.config2(seed=5, target_leaf=40_000, extra=3)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    rng = np.random.default_rng(3)
    f, g, h = (rng.lognormal(40, 2, (p.nblk, 20, 20)) for _ in range(3))
    v = rng.standard_normal((p.nblk, 2, 21, 21)) * 1e6
    tr, lib, out = mg.Transport(**MINIMAL), mg.lib(), []
    for by, blk in ((0, True), (1, True), (0, False)):
        a, b, c, w = shifted(f, by), shifted(g, by), shifted(h * 1e-20, by), shifted(v, by)
        md = shifted(np.full(p.nblk, np.inf), by)
        mn = torch.zeros(1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        if kernel == "netcharge":
            mg.netcharge(ctx, c, a, b)
            res = [c]
        elif kernel == "electric_field":
            mg.electric_field(ctx, w, b, c, p.h1, (1e2, 1e6))
            res = [w, b]
        elif kernel == "flux":
            ctx.check(lib.srmg_streamer_flux_dev(ctx.handle, w.data_ptr(), md.data_ptr() if blk else None, mn.data_ptr(),
                                                 a.data_ptr(), shifted(v, by).data_ptr(), b.data_ptr(), p.nblk, p.h1,
                                                 ctypes.byref(tr)))
            res = [w, mn]
        else:
            ctx.check(lib.srmg_streamer_rates_dev(ctx.handle, a.data_ptr(), c.data_ptr(), shifted(f, by).data_ptr(),
                                                  b.data_ptr(), w.data_ptr(), p.nblk, p.h1, 1, ctypes.byref(tr)))
            res = [a, c]
        ctx.synchronize()
        torch.cuda.synchronize()
        out.append([r.cpu().numpy().copy() for r in res])
    for other in out[1:]:
        for x, y in zip(out[0], other):
            np.testing.assert_array_equal(x.view(np.uint64), y.view(np.uint64))
    ctx.close()
