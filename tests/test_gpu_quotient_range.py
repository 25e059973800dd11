"""Quotients by the cell size of a level whose own size is below the range that the reciprocal is
formed for on level 1: electric_field! (src/multigrid.jl:421-449) on a tree of 30 levels, where
some of them overflow, equals the plain division's bit for bit."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("h", [1.1e-90, 1e-3, 0.9e90])
def test_electric_field_overflows_as_the_division(h):
    import torch
    tree = t2.Tree((1, 1), 30)
    t2.populate(tree, 2)
    for l in range(2, 30):
        t2.refine_block(tree, l, (1, 1))
    tree.sync()
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: 0.0 * r, h)
    rng = np.random.default_rng(4)
    u = rng.choice([-1.0, 1.0], p.b.shape) * 10.0 ** rng.uniform(-310, 308, p.b.shape)
    u[:, ::3] = rng.choice([-1.0, 1.0], u[:, ::3].shape) * 10.0 ** rng.uniform(205, 212, u[:, ::3].shape)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    e = torch.zeros((p.nblk, 2, 21, 21), dtype=torch.float64, device="cuda")
    ug = torch.from_numpy(u).cuda()
    mg.electric_field(ctx, e, torch.zeros_like(ug), ug, h, (0.0, 0.0))
    ctx.synchronize()
    got, overflowed = e.cpu().numpy(), 0
    with np.errstate(over="ignore"):
        for l, layer in enumerate(p.tree, 1):
            for blk in layer.index.values():
                t = u[blk - 1]  # [y, x]
                want = (t[2:18, 1:17] - t[2:18, 2:18]) / (h / 2.0 ** (l - 1)) + 0.0
                overflowed += np.isinf(want).sum()
                np.testing.assert_array_equal(got[blk - 1, 0, 2:18, 2:18].copy().view(np.uint64), want.view(np.uint64))
    assert h > 1e-4 or overflowed > 0
    ctx.close()
