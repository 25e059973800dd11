"""V-cycles with one sweep on level 1 in the persistent kernel, level 1 of several blocks: the sweep's
right-hand side reads the neighbours' restricted residual, which the correction takes the place
of only after all blocks are done.  With one CTA, a few or all of them, and either CTA size, equal
to the per-operation launches bit for bit; solves do not depend on the shape."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

SHAPES = [(0, 768), (0, 1024), (1, 768), (3, 1024), (40, 768)]  # CTAs (0: one an SM), threads


def problem(root, level):
    tree = t2.Tree(root, level)
    t2.populate(tree, level)
    return gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)


@pytest.mark.parametrize("root,level", [((2, 1), 2), ((2, 2), 3), ((5, 3), 2), ((17, 5), 2)])
def test_one_sweep_on_level_1(root, level):
    import torch
    p, out = problem(root, level), []
    start = np.random.default_rng(5).standard_normal(p.b.shape)
    for engine, (ctas, threads) in [(0, (0, 0))] + [(1, s) for s in SHAPES]:
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_option("coarse_cluster", 0).set_option("engine", engine)
        ctx.set_option("engine_ctas", ctas).set_option("engine_threads", threads)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        for l in range(1, level + 1):
            mg.fill_ghost_(ctx, u, l, p.bc)
        mg.vcycle_(ctx, u, b, r, u1, p.s, p.geom, p.bc, None, ndown=2, ntop=1, nup=1, ncycles=3)
        ctx.synchronize()
        out.append([f.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64) for f in (u, b)])
        ctx.close()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("mode", ["MODE_FP64", "MODE_MIXED"])
def test_solves_with_one_sweep(mode):
    import torch
    p, out = problem((5, 3), 2), []  # 15 root blocks: no direct coarsest solve
    for ctas, threads in SHAPES:
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_option("engine_ctas", ctas).set_option("engine_threads", threads)
        b = torch.from_numpy(p.b).cuda()
        u = torch.zeros_like(b)
        mg.solve(ctx, u, b, p.s, p.geom, p.bc, tol=1e-30, mode=getattr(mg, mode), max_cycles=6, ndown=1, ntop=1, nup=1)
        out.append(u.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64))
        ctx.close()
    for u in out[1:]:
        np.testing.assert_array_equal(u, out[0])
