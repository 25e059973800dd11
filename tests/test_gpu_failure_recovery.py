"""A barrier timeout is reported once: calls that follow it on the same context and launch no
persistent kernel of their own (V-cycles and FMG of a tree that fits the coarse cluster) return
SRMG_OK.  The failure is a bounded barrier wait that runs out (no fault, no hang)."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def test_cluster_cycles_after_a_timeout():
    import torch
    tree = t2.Tree((1, 1), 4)
    t2.populate(tree, 4)
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    b = torch.from_numpy(p.b).cuda()
    u, r, u1 = (torch.zeros_like(b) for _ in range(3))
    torch.cuda.synchronize()
    for call in (mg.vcycle_, mg.fmg_):
        assert mg.lib().srmg_selftest_barrier_timeout(ctx.handle, 20) == mg.SRMG_ERR_TIMEOUT
        call(ctx, u, b, r, u1, p.s, p.geom, p.bc, ndown=2, ntop=4, nup=2)
        ctx.synchronize()  # raises unless SRMG_OK
    uh, bh, z = np.zeros_like(p.b), p.b.copy(), np.zeros_like(p.b)
    assert mg.lib().srmg_selftest_barrier_timeout(ctx.handle, 20) == mg.SRMG_ERR_TIMEOUT
    mg.vcycle_(ctx, uh, bh, z.copy(), z.copy(), p.s, p.geom, p.bc, ndown=2, ntop=4, nup=2)
    assert np.isfinite(u.cpu().numpy()).all() and np.isfinite(uh).all()
    ctx.close()
