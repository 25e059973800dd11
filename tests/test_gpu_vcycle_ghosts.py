"""After a V-cycle (src/multigrid.jl:60-106) every level's ghosts are what fill_ghost! makes of the
fields, bit for bit, whichever kernels ran it: the coarse cluster, alone and as the end of the
fused launches or of the persistent kernel, the fused launches of box trees and of octrees.  Among
them trees whose boundary ghosts mirror refinement ghosts.  From a start whose ghosts are filled
the cells do not depend on the path either: the cluster's equal the persistent kernel's."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, gen3, multigrid as mg
from srmg import tree as t2
from srmg import tree3 as t3

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def refined(root, level, towards, box):
    tree = t2.Tree(root, level + len(towards))
    t2.populate(tree, level)
    for k, c in enumerate(towards):
        t2.refine_block(tree, level + k, c, t2.BOX2 if box else t2.STAR2)
    tree.sync()
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)
    return p, t2.connectivity(tree, t2.BOX2) if box else p.conn


def mirrors_refinement(tree):
    """A block at the lower z boundary whose neighbour along r is missing on its level: the corner
    there mirrors the refinement ghosts of that face."""
    return any(c[1] == 1 and layer.in_domain((c[0] + 1, 1)) and (c[0] + 1, 1) not in layer.index
               for layer in list(tree)[1:] for c in layer.index)


TREES = [  # root, uniform levels, blocks refined above them
    ((1, 1), 5, ()),
    ((1, 1), 2, ((1, 1), (2, 2), (3, 3))),
    ((2, 1), 3, ((3, 1), (5, 1))),
    ((1, 1), 6, ()),
    ((1, 1), 5, ((3, 1), (6, 1))),
]


@pytest.mark.parametrize("root,level,towards", TREES)
@pytest.mark.parametrize("lpl", [None, "laplacian4"])
def test_ghosts_are_filled(root, level, towards, lpl):
    import torch
    p, conn = refined(root, level, towards, lpl is not None)
    assert not towards or mirrors_refinement(p.tree)
    start, out = np.random.default_rng(9).standard_normal(p.b.shape), []
    for on in (1, 0):
        ctx = mg.Context(0).set_tree(p.tree, conn)
        ctx.set_option("coarse_cluster", on)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        for l in range(1, len(p.tree) + 1):
            mg.fill_ghost_(ctx, u, l, p.bc)
        mg.vcycle_(ctx, u, b, r, u1, p.s, gen.GEOM_CYL1, p.bc, lpl, ndown=2, ntop=4, nup=2, ncycles=2)
        ctx.synchronize()
        got = u.cpu().numpy()
        for l in range(1, len(p.tree) + 1):
            mg.fill_ghost_(ctx, u, l, p.bc)
        ctx.synchronize()
        np.testing.assert_array_equal(got.view(np.uint64), u.cpu().numpy().view(np.uint64))
        out.append((got, b.cpu().numpy()[:, 2:18, 2:18].copy()))
        ctx.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x.view(np.uint64), y.view(np.uint64))


@pytest.mark.parametrize("stencil,lpl", [("star", "laplacian"), ("box", "laplacian"), ("box", "laplacian4")])
def test_ghosts_are_filled_octree(stencil, lpl):
    import torch
    tree = t3.Tree3((1, 1, 1), 4)
    t3.populate(tree, 2)
    for l in (2, 3):
        t3.refine_block(tree, l, (1, 1, 1), t3.BOX3)
    tree.sync()
    conn = t3.connectivity(tree, t3.BOX3 if stencil == "box" else t3.STAR3)
    s = (1.0 / 16) ** 2
    p = gen3.make_problem3(tree, conn, lambda x, y, z: np.cos(3 * x) * y * (1 - z), s)
    bc = t3.boundaryconditions(((-1, -1), (1, -1), (-1, 1)))
    ctx = mg.Context(0, D=3).set_tree(tree, conn)
    b = torch.from_numpy(p.b).cuda()
    u = torch.from_numpy(np.random.default_rng(9).standard_normal(p.b.shape)).cuda()
    r, u1 = torch.zeros_like(b), torch.zeros_like(b)
    for l in range(1, 5):
        mg.fill_ghost_(ctx, u, l, bc)
    mg.vcycle_(ctx, u, b, r, u1, s, 0, bc, lpl, ndown=2, ntop=4, nup=2)
    ctx.synchronize()
    got = u.cpu().numpy()
    for l in range(1, 5):
        mg.fill_ghost_(ctx, u, l, bc)
    ctx.synchronize()
    np.testing.assert_array_equal(got.view(np.uint64), u.cpu().numpy().view(np.uint64))
    ctx.close()
