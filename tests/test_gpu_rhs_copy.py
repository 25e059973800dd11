"""rhs_level! of order 2 (src/multigrid.jl:363-388, the identity on the valid cells) by pairs of cells
where both fields start on 16 bytes, else cell by cell: the same cells, no ghost written."""
import numpy as np
import pytest

from conftest import gpu_available
from srmg import gen, multigrid as mg

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("shift_in,shift_out", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_copy_of_the_valid_cells(shift_in, shift_out):
    import torch
    p = gen.config2(seed=5, target_leaf=40_000, extra=3)
    ctx = mg.Context(0).set_tree(p.tree, p.conn)
    a = np.random.default_rng(2).standard_normal(p.b.shape)

    def placed(x, by):
        t = torch.zeros(x.size + 2, dtype=torch.float64, device="cuda")[by:by + x.size].view(*x.shape)
        return t.copy_(torch.from_numpy(x))

    q, out = placed(a, shift_in), placed(np.full_like(a, -3.0), shift_out)
    torch.cuda.synchronize()
    want = np.full_like(a, -3.0)
    for l, layer in enumerate(p.tree, 1):
        mg.rhs_level_(ctx, out, q, l, p.geom)
        for k in layer.index.values():
            want[k - 1, 2:18, 2:18] = a[k - 1, 2:18, 2:18]
    ctx.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want.view(np.uint64))
    ctx.close()
