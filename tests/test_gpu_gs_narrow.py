"""Which single-process sweeps run in one block: decided by the warps that a
level keeps busy (up to 8), so by the call's width as well as by the schedule.
27-point operators, items of eight rows: one warp each up to 64 bytes a row, two
and four beyond.  The whole device takes two launches a call (a sweep each), one
block takes one."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,prec,nv,launches", [
    (16, 0, 8, 1), (16, 0, 16, 2), (16, 0, 32, 2), (16, 1, 16, 1), (16, 1, 32, 2),  # 5.1 items a level
    (12, 0, 16, 1), (12, 0, 32, 2), (12, 1, 32, 1),                                 # 3.3 items a level
    (24, 0, 1, 2),                                                                  # 11 items a level
])
def test_block_or_device(gpu, side, prec, nv, launches):
    d = sp.diags([np.ones(side - 1), np.ones(side), np.ones(side - 1)], [-1, 0, 1])
    A = (27.0 * sp.identity(side ** 3) - 0.5 * sp.kron(sp.kron(d, d), d)).tocsr()
    A.sort_indices()
    n, dtype = A.shape[0], np.float64 if prec == 0 else np.float32
    rp, ci, v = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    L = xamg.lib()
    plan = L.xamg_gs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), 0, 1)
    assert plan
    try:
        xamg.check(L.xamg_gs_plan_set_values(plan, xamg._ptr(v), prec))
        rng = np.random.default_rng(1)
        h = [rp, ci, v.astype(dtype), np.full(n, 1 / 26.5, dtype), rng.uniform(-1, 1, (n, nv)).astype(dtype),
             np.zeros((n, nv), dtype), np.ones(nv, dtype)]
        t = [torch.as_tensor(a).cuda() for a in h]
        torch.cuda.synchronize()
        before = L.XAMG_b200_kernel_launches()
        xamg.check(L.xamg_hsgs(plan, prec, nv, *[a.data_ptr() for a in t], None, None))
        torch.cuda.synchronize()
        assert L.XAMG_b200_kernel_launches() - before == launches
        assert L.xamg_gs_plan_error(plan) == 0
    finally:
        L.xamg_gs_plan_destroy(plan)
