"""The octree sweep that writes its ghosts by rule and loads its faces ahead of its wait (star
connectivity, order 2) and the fused steps around it against other bodies: the V-cycle recorded
for the sequencer, whose sweeps are the plain grid-stride loop (option `gs_push` 0 changes
the steps around the sweeps only).  Cells bit for bit, from a start whose ghosts are not filled."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen3, multigrid as mg, tree3 as t3

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

BC = t3.boundaryconditions(((-1, -1), (1, -1), (-1, 1)))
CASES = [((1, 1, 1), 1, ()), ((1, 2, 1), 2, ()), ((1, 1, 1), 2, ((1, 1, 1), (2, 2, 2))), ((1, 1, 1), 3, ((3, 2, 3),))]


def problem(root, level, towards, lpl):
    tree = t3.Tree3(root, level + len(towards))
    t3.populate(tree, level)
    for k, c in enumerate(towards):
        t3.refine_block(tree, level + k, c, t3.BOX3)
    tree.sync()
    return gen3.make_problem3(tree, t3.connectivity(tree, t3.STAR3), lambda x, y, z: np.cos(3 * x) * y * (1 - z),
                              (1.0 / 16) ** 2)


@pytest.mark.parametrize("root,level,towards", CASES)
@pytest.mark.parametrize("lpl", ["laplacian", ("helmholtz", 30.0)])
def test_vcycle_against_the_sequencer(root, level, towards, lpl):
    import torch
    p, out = problem(root, level, towards, lpl), []
    start = np.random.default_rng(11).standard_normal(p.b.shape)
    for sequencer in (0, 1):
        ctx = mg.Context(0, D=3).set_tree(p.tree, p.conn)
        ctx.set_option("op_graphs", 0).set_option("op_sequencer", sequencer)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        torch.cuda.synchronize()
        before = ctx.launches()
        mg.vcycle_(ctx, u, b, r, u1, p.s, 0, BC, lpl, ndown=2, ntop=4, nup=2, ncycles=2)
        launches = ctx.launches() - before
        ctx.synchronize()
        assert (launches == 1) == bool(sequencer)
        out.append([f.cpu().numpy()[(slice(None),) + (slice(2, 18),) * 3].copy().view(np.uint64) for f in (u, b)])
        ctx.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
