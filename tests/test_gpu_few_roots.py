"""Trees whose level 1 has two to four blocks, which one CTA of the persistent kernel works on: the
V-cycle's fields and every solve do not depend on how many blocks a CTA takes at a time (option
`engine_threads`: 768 threads are three, 1024 four), trees of a single level among them, whose
next phase is every CTA's; V-cycles equal the per-operation launches bit for bit."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

ROOTS = [(2, 1), (1, 3), (2, 2), (4, 1), (1, 4)]


def problem(root, level):
    tree = t2.Tree(root, level)
    t2.populate(tree, level)
    return gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)


@pytest.mark.parametrize("root", ROOTS)
@pytest.mark.parametrize("level", [1, 2, 3])
@pytest.mark.parametrize("ntop", [3, 4])
def test_vcycle_equals_the_launches(root, level, ntop):
    import torch
    p, out = problem(root, level), []
    start = np.random.default_rng(5).standard_normal(p.b.shape)
    for engine, threads in ((0, 0), (1, 768), (1, 1024)):
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_option("coarse_cluster", 0).set_option("engine", engine).set_option("engine_threads", threads)
        for _ in range(1 if not engine else 4):
            b = torch.from_numpy(p.b).cuda()
            u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
            for l in range(1, level + 1):
                mg.fill_ghost_(ctx, u, l, p.bc)
            mg.vcycle_(ctx, u, b, r, u1, p.s, p.geom, p.bc, None, ndown=1, ntop=ntop, nup=2, ncycles=2)
            ctx.synchronize()
            out.append([f.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64) for f in (u, b)])
        ctx.close()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("root", [(1, 3), (2, 2)])
@pytest.mark.parametrize("level", [1, 2, 3])
@pytest.mark.parametrize("mode", ["MODE_MIXED", "MODE_FP64_DIRECT", "MODE_FP64"])
@pytest.mark.parametrize("direct_level", [0, 1])
def test_solves_do_not_depend_on_the_shape(root, level, mode, direct_level):
    import torch
    p, out = problem(root, level), []
    for threads in (768, 1024):
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_option("engine_threads", threads).set_option("direct_level", direct_level)
        b = torch.from_numpy(p.b).cuda()
        for _ in range(3):
            u = torch.zeros_like(b)
            # the reference's cycle (MODE_FP64) contracts slowly on 16 x 64 cells: thirty of them
            st = mg.solve(ctx, u, b, p.s, p.geom, p.bc, tol=1e-9, mode=getattr(mg, mode),
                          max_cycles=30 if mode == "MODE_FP64" else 400)
            assert mode == "MODE_FP64" or st["rel_residual"] <= 1e-9, st
            out.append((st["cycles"], u.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64)))
        norm = mg.resnorm(ctx, None, b, u, p.s, p.geom, p.bc)
        scale = mg.resnorm(ctx, None, b, torch.zeros_like(b), p.s, p.geom, p.bc)
        assert mode == "MODE_FP64" or norm <= 1.0001e-9 * scale
        ctx.close()
    for c, u in out[1:]:
        assert c == out[0][0]
        np.testing.assert_array_equal(u, out[0][1])
