"""The free-boundary transforms of one CTA at every count of radix-2 stages left over by its
four-stage passes, n = 16 (one pass) to 8192 (its largest), against the oracle's FFTs (src/freebc.jl:
93-102): both round to a few ulp of the largest term, 1e-12 relative as in test_gpu_freebc."""
import numpy as np
import pytest

import freebc_oracle as fo
from conftest import gpu_available
from srmg import gen, multigrid as mg, tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("level", [1, 2, 3, 4, 5, 6, 7, 8, 10])
def test_freebc_every_length(level):
    import torch
    tree = t2.Tree((1, 1), min(level, 2))
    t2.populate(tree, min(level, 2))
    p = gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj), 1e-4)
    n, H, R, f = fo.kernel(1, level, (1, 1), p.h1)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    mg.freebc_set(ctx, 1, level, (1, 1), f)
    rng = np.random.default_rng(level)
    u, q = rng.standard_normal(p.b.shape), rng.standard_normal(p.b.shape)
    qg, ug = torch.from_numpy(q).cuda(), torch.from_numpy(u).cuda()
    bg = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    mg.freebc_(ctx, qg, ug, p.h1, p.s, b_out=bg)
    ctx.synchronize()
    qo = q.copy()
    bo = fo.freebc(qo, u, p.h1, p.s, p.tree, p.conn, 1, level, f)
    got, changed = qg.cpu().numpy(), qo != q
    assert np.linalg.norm(bg.cpu().numpy() - bo) <= 1e-12 * np.linalg.norm(bo)
    assert np.array_equal(got[~changed], q[~changed])
    assert np.linalg.norm((got - qo)[changed]) <= 1e-12 * np.linalg.norm((qo - q)[changed]) + 1e-15 * np.linalg.norm(q)
    ctx.close()
