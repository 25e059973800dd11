"""The fused V-cycle of octrees (src/multigrid.jl:42-106 with D = 3): residual and restriction in one
pass, the saved level with the coarse right-hand side, the filled correction, the prolongation
and the sweeps writing their ghosts.  Bit for bit the unfused launches (option `gs_push` 0), on
single blocks, uniform and refined trees (refined at a corner of the domain too, where boundary
ghosts mirror refinement ghosts), star and box connectivity, from a start whose ghosts are not
filled."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen3, multigrid as mg, tree3 as t3

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def octree(root, level, towards):
    tree = t3.Tree3(root, level + len(towards))
    t3.populate(tree, level)
    for k, c in enumerate(towards):
        t3.refine_block(tree, level + k, c, t3.BOX3)
    tree.sync()
    return tree


CASES = [  # root blocks, uniform levels, blocks refined above them, stencil, operator, lmax, sweeps
    ((1, 1, 1), 1, (), "star", "laplacian", 0, (2, 4, 2)),
    ((1, 2, 1), 2, (), "star", ("helmholtz", 30.0), 0, (1, 1, 1)),
    ((1, 1, 1), 2, ((1, 1, 1), (2, 2, 2)), "star", "laplacian", 0, (2, 3, 1)),
    ((1, 1, 1), 3, ((3, 2, 3),), "star", "laplacian", 3, (2, 4, 2)),
    ((1, 1, 1), 2, ((1, 1, 1), (1, 1, 1), (1, 2, 1)), "box", "laplacian4", 0, (2, 4, 2)),
    ((2, 1, 1), 2, ((3, 2, 1),), "box", "laplacian4", 0, (1, 2, 3)),
    ((1, 1, 1), 2, ((2, 1, 2),), "box", "laplacian", 0, (2, 4, 2)),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[3]}_{c[4]}_{c[0]}_{len(c[2])}")
def test_vcycle_fused_bit_identical(case):
    import torch
    root, level, towards, stencil, lpl, lmax, (nd, nt, nu) = case
    tree = octree(root, level, towards)
    conn = t3.connectivity(tree, t3.BOX3 if stencil == "box" else t3.STAR3)
    s = (1.0 / 16) ** 2
    p = gen3.make_problem3(tree, conn, lambda x, y, z: np.cos(3 * x) * y * (1 - z), s)
    bc = t3.boundaryconditions(((-1, -1), (1, -1), (-1, 1)))
    start = np.random.default_rng(11).standard_normal(p.b.shape)
    v = (slice(None),) + (slice(2, 18),) * 3
    out = {}
    for push in (1, 0):
        ctx = mg.Context(0, D=3).set_tree(tree, conn)
        ctx.set_option("gs_push", push)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        torch.cuda.synchronize()
        mg.vcycle_(ctx, u, b, r, u1, s, 0, bc, lpl, lmax=lmax, ndown=nd, ntop=nt, nup=nu, ncycles=2)
        ctx.synchronize()
        out[push] = (u.cpu().numpy()[v].copy(), b.cpu().numpy()[v].copy())
        ctx.close()
    for a, g, what in zip(out[1], out[0], ("u", "b")):
        np.testing.assert_array_equal(a.view(np.uint64), g.view(np.uint64), err_msg=what)
