"""Tables of the coarse cluster belong to the tree: several trees on one context, one after the
other on a stream of the caller's, V-cycles (src/multigrid.jl:60-106) launched right after the
upload, give what the per-operation launches of a fresh context give, bit for bit."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def uniform(root, level):
    tree = t2.Tree(root, level)
    t2.populate(tree, level)
    return gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)


def cycle(ctx, p, lpl, start, stream):
    """One V-cycle from a start with filled ghosts; the fields, still in flight."""
    import torch
    with torch.cuda.stream(stream):
        u, b = torch.from_numpy(start).cuda(), torch.from_numpy(p.b).cuda()
        r, u1 = torch.zeros_like(b), torch.zeros_like(b)
        for l in range(1, len(p.tree) + 1):
            mg.fill_ghost_(ctx, u, l, p.bc)
        mg.vcycle_(ctx, u, b, r, u1, p.s, p.geom, p.bc, lpl, ndown=2, ntop=4, nup=2)
    return u, b, r, u1


def test_trees_in_turn():
    import torch
    probs = [(uniform((1, 1), 5), None), (gen.config2(seed=5, target_leaf=60_000, base_level=3, extra=3), None),
             (gen.order4_problem(seed=62, geom=1, base_level=4, extra=2), "laplacian4"), (uniform((17, 1), 3), None),
             (uniform((1, 1), 5), None)]
    starts = [np.random.default_rng(k).standard_normal(p.b.shape) for k, (p, _) in enumerate(probs)]
    stream = torch.cuda.Stream()
    one, got = mg.Context(0), []
    one.set_stream(stream.cuda_stream)
    for (p, lpl), start in zip(probs, starts):
        one.set_tree(p.tree, p.conn)
        got.append(cycle(one, p, lpl, start, stream))
    one.synchronize()
    for k, ((p, lpl), start) in enumerate(zip(probs, starts)):
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_stream(stream.cuda_stream)
        ctx.set_option("coarse_cluster", 0).set_option("engine", 0).set_option("gs_push", 0)
        want = cycle(ctx, p, lpl, start, stream)
        ctx.synchronize()
        for a, g, what in zip(got[k], want, "ub"):
            a, g = (x.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64) for x in (a, g))
            np.testing.assert_array_equal(a, g, err_msg=f"tree {k}, {what}")
        ctx.close()
    one.close()
