"""The coarse cluster's tables are an aid: where the device has no memory left for them, a V-cycle
runs without them and gives the same values."""
import ctypes

import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg
from srmg import tree as t2

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def uniform(level):
    tree = t2.Tree((1, 1), level)
    t2.populate(tree, level)
    return gen.make_problem(tree, lambda r, z, l, gi, gj: gen.cell_hash01(3, l, gi, gj) - 0.5, 1e-4)


def test_vcycle_without_memory_for_the_tables():
    import torch
    small, p = uniform(1), uniform(5)
    b = torch.from_numpy(p.b).cuda()
    fields = [[torch.zeros_like(b), b.clone(), torch.zeros_like(b), torch.zeros_like(b)] for _ in range(2)]
    rt = ctypes.CDLL("libcudart.so.12")
    ctx = mg.Context(0).set_tree(small.tree, small.conn)

    def cycle(f, q):
        torch.cuda.synchronize()
        mg.vcycle_(ctx, *f, q.s, q.geom, q.bc, ndown=2, ntop=4, nup=2)
        ctx.synchronize()

    cycle([torch.zeros(small.b.shape, dtype=torch.float64, device="cuda") for _ in range(4)], small)
    ctx.set_tree(p.tree, p.conn)
    ctx.set_option("coarse_cluster", 0)
    cycle(fields[0], p)  # every other buffer of a cycle exists now
    ctx.set_option("coarse_cluster", 1)
    held = []
    try:
        size = 1 << 36
        while size >= 1 << 12:
            q = ctypes.c_void_p()
            if rt.cudaMalloc(ctypes.byref(q), ctypes.c_size_t(size)) == 0:
                held.append(q)
            else:
                size >>= 1
        rt.cudaGetLastError()
        cycle(fields[1], p)
    finally:
        for q in held:
            rt.cudaFree(q)
    for x, y in zip(fields[0][:2], fields[1][:2]):
        x, y = (t.cpu().numpy()[:, 2:18, 2:18].copy().view(np.uint64) for t in (x, y))
        np.testing.assert_array_equal(x, y)
    ctx.close()
