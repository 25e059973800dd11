"""Quotients by a fixed divisor through its reciprocal equal the division bit for bit (the residual
-(b + L(u) / s) of a level, src/multigrid.jl:349-354, against the oracle's): stencil values that
are zeros of either sign, subnormal, close to the largest double, infinite or NaN, and level
scales from tiny (where the division itself is taken) to large."""
import ctypes
import dataclasses

import numpy as np
import pytest

from conftest import gpu_available
from oracle import Oracle, lib as olib, _ptr
from srmg import gen, multigrid as mg

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("s", [1e-300, 3e-91, 1.7e-16, -0.3, 1.0, 7.0, 1e80, 1e95])
def test_residual_at_the_ends_of_the_range(s):
    import torch
    p = gen.order4_problem(seed=53, geom=gen.GEOM_CYL1)
    for lpl_op in (0, 2):
        orc = Oracle(dataclasses.replace(p, op=lpl_op))
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        rng = np.random.default_rng(9)
        u = rng.standard_normal(p.b.shape) * 10.0 ** rng.uniform(-320, 300, p.b.shape)
        u[rng.random(u.shape) < 0.3] = 0.0
        u[rng.random(u.shape) < 0.3] *= -1.0
        u[0, 5, 5], u[0, 9, 9], u[1, 7, 7] = np.inf, np.nan, -np.inf
        b = np.where(rng.random(u.shape) < 0.5, -0.0, rng.standard_normal(u.shape))
        ug, bg = torch.from_numpy(u).cuda(), torch.from_numpy(b).cuda()
        rg = torch.zeros_like(bg)
        torch.cuda.synchronize()
        ro = np.zeros_like(u)
        for l in range(1, len(p.tree) + 1):
            ctx.check(mg.lib().srmg_residual_level_dev(ctx.handle, rg.data_ptr(), ug.data_ptr(), bg.data_ptr(), p.nblk, l,
                                                       s, lpl_op, 0.0, p.geom))
            olib().orc_residual_level(_ptr(ro), _ptr(u), _ptr(b), s, orc.ot.ref, l, ctypes.byref(orc.op))
        ctx.synchronize()
        got = rg.cpu().numpy()
        nan = np.isnan(ro)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got[~nan].view(np.uint64), ro[~nan].view(np.uint64))
        ctx.close()
