"""The coarse levels of an FP64 V-cycle in one cluster (option `coarse_cluster`, on by
default): V-cycles and FMG (src/multigrid.jl:42-106) equal those of the launches and of the
persistent kernel bit for bit -- every step forms each value by the same operations in the same
order -- where the whole tree fits in the cluster and where it is its coarse end; one block,
one more than a CTA each, a full share of every CTA; refined levels, box trees, every geometry,
sweep counts that leave a level in the persistent kernel's second buffer.  The start's ghosts
are not filled: where the whole cycle runs in the cluster its partner is the per-operation
path, which reads them as the reference does (the persistent kernel takes a neighbour's cells
from them).  FMG fills them first; there the partner is the default path."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

BC = {gen.GEOM_CART: t2.boundaryconditions(((-1, -1), (-1, -1))), gen.GEOM_CYL1: gen.BC_POISSON,
      gen.GEOM_CYL2: t2.boundaryconditions(((-1, 1), (1, 1)))}


def uniform(root, level):
    tree = t2.Tree(root, level)
    t2.populate(tree, level)
    return gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)


# name, problem, operator, geometry, lmax (0: all), sweeps, options, whether it fits whole
def cases():
    one = uniform((1, 1), 6)
    for lmax, sweeps, geom in ((1, (2, 4, 2), 1), (2, (1, 1, 1), 0), (5, (2, 4, 2), 2), (6, (3, 5, 2), 1),
                               (6, (2, 4, 2), 0)):
        yield f"uniform_{lmax}", one, None, geom, lmax, sweeps, {}, lmax <= 5
    yield "roots_17", uniform((17, 1), 3), None, 1, 2, (1, 2, 3), {}, True
    yield "roots_15", uniform((3, 5), 4), ("helmholtz", 2e3), 2, 3, (2, 4, 2), {}, True
    yield "engine_off", one, ("helmholtz", 2e3), 1, 6, (2, 3, 1), {"engine": 0}, False
    for leaf, base, geom in ((20_000, 2, 1), (60_000, 3, 0), (200_000, 5, 1)):
        p = gen.config2(seed=5, target_leaf=leaf, base_level=base, extra=3)
        yield f"channel_{leaf}", p, None, geom, 0, (2, 4, 2), {}, leaf <= 60_000
    for geom in (0, 1, 2):
        p = gen.order4_problem(seed=61 + geom, geom=geom, base_level=4, extra=2)
        yield f"box_order4_{geom}", p, "laplacian4", geom, 0, (2, 4, 2), {}, False
    yield "box_order2", p, None, 2, 0, (1, 4, 1), {}, False


@pytest.mark.parametrize("case", list(cases()), ids=lambda c: c[0])
def test_vcycle_and_fmg_coarse_levels_bit_identical(case):
    import torch
    _, p, lpl, geom, lmax, (nd, nt, nu), opts, whole = case
    bc = BC[geom] if "box" not in case[0] else p.bc
    start = np.random.default_rng(7).standard_normal(p.b.shape)  # ghosts too: a fill comes first
    out = {}
    for on in (1, 0):
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        for k, v in dict(opts, coarse_cluster=on).items():
            ctx.set_option(k, v)
        if not on and whole:
            ctx.set_option("engine", 0)
        b = torch.from_numpy(p.b).cuda()
        u, r, u1 = torch.from_numpy(start).cuda(), torch.zeros_like(b), torch.zeros_like(b)
        torch.cuda.synchronize()
        mg.vcycle_(ctx, u, b, r, u1, p.s, geom, bc, lpl, lmax=lmax, ndown=nd, ntop=nt, nup=nu, ncycles=2)
        ctx.synchronize()
        got = [u.cpu().numpy().copy(), b.cpu().numpy().copy()]
        if not on and whole:
            ctx.set_option("engine", opts.get("engine", 1))
        u.zero_()
        b.copy_(torch.from_numpy(p.b))
        torch.cuda.synchronize()
        mg.fmg_(ctx, u, b, r, u1, p.s, geom, bc, lpl, ndown=nd, ntop=nt, nup=nu)
        ctx.synchronize()
        out[on] = got + [u.cpu().numpy().copy()]
        ctx.close()
    v = (slice(None), slice(2, 18), slice(2, 18))
    for a, g, what in zip(out[1], out[0], ("vcycle u", "vcycle b", "fmg u")):
        np.testing.assert_array_equal(a[v].copy().view(np.uint64), g[v].copy().view(np.uint64), err_msg=what)
