"""Block sweeps with a level of more items than an mbarrier can count arrivals
for (2^20 - 1): a diagonal matrix of two blocks, whose rows are all of one
level.  FP64, NV 32: a warp holds two rows of an item of eight, so an item
arrives four times.  One row fewer than the limit's items, and beyond it."""
import numpy as np
import pytest
import torch

import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("brows", [8 * (2 ** 18 - 1), 8 * 2 ** 18 + 8])
def test_one_level(gpu, brows):
    n, nv = brows + 1000, 32
    L = xamg.lib()
    rng = np.random.default_rng(3)
    rp, ci = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    v = np.full(n, 2.0)  # a power of two: the sweep's sums are exact
    plan = L.xamg_gs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), brows, 1)
    assert plan
    try:
        xamg.check(L.xamg_gs_plan_set_values(plan, xamg._ptr(v), 0))
        small = torch.as_tensor(rng.integers(-8, 8, n).astype(np.float64)).cuda()
        b = small[:, None] + torch.arange(nv, dtype=torch.float64, device="cuda")
        x = torch.ones((n, nv), dtype=torch.float64, device="cuda")
        t = torch.zeros_like(b)
        keep = [torch.as_tensor(a).cuda() for a in (rp, ci, v, np.full(n, 0.5), np.full(nv, 0.5))]
        q = [a.data_ptr() for a in (keep[0], keep[1], keep[2], keep[3], b, x, keep[4], t)]
        torch.cuda.synchronize()
        xamg.check(L.xamg_hsgs(plan, 0, nv, *q, None))
        torch.cuda.synchronize()
        # twice x += 0.5 * 0.5 * (b - 2 x)
        y = torch.ones_like(x)
        for _ in range(2):
            y += 0.25 * (b - 2 * y)
        assert torch.equal(x, y)
        assert L.xamg_gs_plan_error(plan) == 0
    finally:
        L.xamg_gs_plan_destroy(plan)
