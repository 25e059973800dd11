"""The diffusion time-step limit h_l h_l / D / 4 of flux! (src/fluid.jl) at cell sizes whose
squares leave the range of a double on some levels only: each leaf block's is formed from its
own level's cell size, bit for bit."""
import ctypes

import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2
from srmg.streamer import MINIMAL

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("h", [3e154, 1.6e154, 1e-4, 3e-161, 1e-154])
@pytest.mark.parametrize("D", [0.18, 7e-200])
def test_limit_of_each_block(h, D):
    import torch
    tree = t2.Tree((1, 1), 4)
    t2.populate(tree, 3)
    t2.refine_block(tree, 3, (2, 2))
    tree.sync()
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: 0.0 * r, h)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    ones = torch.ones((p.nblk, 20, 20), dtype=torch.float64, device="cuda")
    still = torch.zeros((p.nblk, 2, 21, 21), dtype=torch.float64, device="cuda")  # no drift: no other limit
    flux, blk = torch.zeros_like(still), torch.full((p.nblk,), -1.0, dtype=torch.float64, device="cuda")
    least = torch.zeros(2, dtype=torch.float64, device="cuda")
    tr = mg.Transport(**dict(MINIMAL, D=D))
    torch.cuda.synchronize()
    for per_block, m in ((blk.data_ptr(), least[:1]), (None, least[1:])):
        ctx.check(mg.lib().srmg_streamer_flux_dev(ctx.handle, flux.data_ptr(), per_block, m.data_ptr(), ones.data_ptr(),
                                                  still.data_ptr(), ones.data_ptr(), p.nblk, h, ctypes.byref(tr)))
    ctx.synchronize()
    blk, least, want = blk.cpu().numpy(), least.cpu().numpy(), []
    with np.errstate(all="ignore"):
        for l, layer in enumerate(p.tree, 1):
            hl = np.float64(h) / 2.0 ** (l - 1)
            for c, k in layer.index.items():
                if p.tree.isleaf(l, c):
                    want.append(np.fmin(np.inf, hl * hl / np.float64(D) / 4.0))
                    assert blk[k - 1] == want[-1], (l, blk[k - 1], want[-1])
    assert (least == min(want)).all()
    ctx.close()
