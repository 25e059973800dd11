"""Net charge, electric field and flux restriction walk the tree's blocks, whatever their ids: with
ids spread over 400 times their number (a pool that a larger tree was freed from) the blocks'
values are those of dense ids bit for bit, other ids' storage is not touched, and a call takes
no longer than the dense one by more than a launch's worth."""
import ctypes

import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg.streamer import MINIMAL
from srmg.tree import connectivity

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

SPREAD = 400


def microseconds(stream, call):
    import torch
    best = np.inf
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(stream)
        call()
        b.record(stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


def test_spread_ids():
    import torch
    tr, lib, stream, out = mg.Transport(**MINIMAL), mg.lib(), torch.cuda.Stream(), []
    rng = np.random.default_rng(3)
    for spread in (1, SPREAD):
        p = gen.config2(seed=5, target_leaf=40_000, extra=3)
        n = p.nblk
        ids = np.arange(n) * spread
        if spread > 1:
            for layer in p.tree:
                layer.index = {c: int(ids[b - 1]) + 1 for c, b in layer.index.items()}
                layer.coord = {b: c for c, b in layer.index.items()}
            p.tree.sync()
            p.conn = connectivity(p.tree)
        else:
            scalar = [rng.lognormal(40, 2, (n, 20, 20)) for _ in range(3)]
            vector = rng.standard_normal((n, 2, 21, 21)) * 1e6
        total, at = int(ids[-1]) + 1, torch.from_numpy(ids).cuda()

        def placed(a):
            t = torch.full((total,) + a.shape[1:], -7.0, dtype=torch.float64, device="cuda")
            t[at] = torch.from_numpy(a).cuda()
            return t

        ne, ni, u = (placed(a) for a in scalar)
        q, eabs, e, flux = placed(scalar[2]), placed(scalar[2]), placed(vector), placed(vector)
        least = torch.zeros(1, dtype=torch.float64, device="cuda")
        ctx = mg.Context(0).set_tree(p.tree, p.conn)
        ctx.set_stream(stream.cuda_stream)
        torch.cuda.synchronize()
        e0 = (ctypes.c_double * 2)(1e2, 1e6)
        calls = [lambda: ctx.check(lib.srmg_netcharge_dev(ctx.handle, q.data_ptr(), ne.data_ptr(), ni.data_ptr(), total)),
                 lambda: ctx.check(lib.srmg_electric_field_dev(ctx.handle, e.data_ptr(), eabs.data_ptr(), u.data_ptr(),
                                                               total, p.h1, ctypes.addressof(e0))),
                 lambda: ctx.check(lib.srmg_streamer_flux_dev(ctx.handle, flux.data_ptr(), None, least.data_ptr(),
                                                              ne.data_ptr(), e.data_ptr(), eabs.data_ptr(), total, p.h1,
                                                              ctypes.byref(tr)))]
        us = [microseconds(stream, c) for c in calls]
        ctx.synchronize()
        fields = (q, eabs, e, flux)
        out.append((us, [f[at].cpu().numpy() for f in fields]))
        for f in fields:
            f[at] = -7.0
            assert bool((f == -7.0).all())
        ctx.close()
    for x, y in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(x.view(np.uint64), y.view(np.uint64))
    for dense, spread in zip(out[0][0], out[1][0]):
        assert spread < 2 * dense + 20, (out[0][0], out[1][0])
