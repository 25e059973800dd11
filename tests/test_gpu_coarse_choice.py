"""Which V-cycles use the coarse cluster: those that its cut makes shorter.  Counted in launches of
the calls on flat trees, where it makes them longer (equal to those with option
`coarse_cluster` 0), and on deep ones, where it does not; the values agree bit for bit."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

# root blocks, levels, operator on box connectivity (None: star, order 2), options, sweeps, cluster used
CASES = [
    ((16, 16), 1, "laplacian4", {}, (2, 4, 2), False),
    ((16, 16), 2, "laplacian4", {}, (2, 4, 2), False),
    ((8, 8), 2, "laplacian4", {}, (1, 1, 1), False),
    ((8, 8), 2, "laplacian4", {}, (2, 4, 2), True),
    ((1, 1), 5, "laplacian4", {}, (2, 4, 2), True),
    ((16, 16), 2, None, {"engine": 0}, (2, 4, 2), False),
    ((1, 1), 5, None, {"engine": 0}, (1, 1, 1), True),
    ((2, 4), 4, None, {}, (1, 1, 1), False),
    ((2, 4), 4, None, {}, (2, 4, 2), True),
    ((1, 3), 5, None, {}, (1, 1, 1), True),
    ((8, 8), 2, None, {}, (1, 1, 1), False),
    ((8, 8), 2, None, {}, (2, 4, 2), True),
    ((1, 1), 5, None, {}, (1, 1, 1), True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}_{c[1]}_{c[2]}_{len(c[3])}_{c[4]}")
def test_launches(case):
    import torch
    root, level, lpl, opts, (nd, nt, nu), used = case
    tree = t2.Tree(root, level)
    t2.populate(tree, level)
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)
    conn = t2.connectivity(tree, t2.BOX2) if lpl else p.conn
    start = np.random.default_rng(5).standard_normal(p.b.shape)
    launches, fields = [], []
    for on in (1, 0):
        ctx = mg.Context(0).set_tree(tree, conn)
        for k, v in dict(opts, coarse_cluster=on, op_graphs=0).items():
            ctx.set_option(k, v)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        for l in range(1, level + 1):
            mg.fill_ghost_(ctx, u, l, p.bc)
        before = ctx.launches()
        mg.vcycle_(ctx, u, b, r, u1, p.s, p.geom, p.bc, lpl, ndown=nd, ntop=nt, nup=nu)
        launches.append(ctx.launches() - before)
        ctx.synchronize()
        fields.append([f.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64) for f in (u, b)])
        ctx.close()
    assert (launches[0] != launches[1]) == used or (used and launches == [1, 1]), launches
    for x, y in zip(*fields):
        np.testing.assert_array_equal(x, y)
