"""Gauss-Seidel sweeps of matrices with a row of more entries than the
level-ordered copy can hold (2^18): such plans take their values and sweep over
the matrix as given, with the oracle's values."""
import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("n,brows", [(270000, 0), (280000, 265000)])
@pytest.mark.parametrize("nv", [1, 4])
def test_dense_row(gpu, n, brows, nv, schedule):
    rng = np.random.default_rng(nv)
    dense = 5
    # row 5 has every column; the others read it
    rows = [np.unique(np.array([dense, i])) for i in range(n)]
    rows[dense] = np.arange(n)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.concatenate(rows).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1])
    v[ci == np.repeat(np.arange(n), np.diff(rp))] = 4.0
    v[rp[dense]:rp[dense + 1]] *= 1e-4
    v[rp[dense] + dense] = 4.0
    invd = np.full(n, 0.25)
    L = xamg.lib()
    plan = L.xamg_gs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), brows, schedule)
    assert plan
    try:
        xamg.check(L.xamg_gs_plan_set_values(plan, xamg._ptr(v), 0))
        b, x0 = rng.uniform(-1, 1, (n, nv)), rng.uniform(-1, 1, (n, nv))
        relax = np.full(nv, 0.99)
        keep = [torch.as_tensor(a).cuda() for a in (rp, ci, v, invd, b, x0, relax, np.zeros_like(b))]
        q = [t.data_ptr() for t in keep]
        torch.cuda.synchronize()
        xamg.check(L.xamg_hsgs(plan, 0, nv, *q[:8], None))
        torch.cuda.synchronize()
        ref = orc.hsgs(rp, ci, v, invd, b, x0.copy(), relax, block_rows=brows)
        assert np.array_equal(keep[5].cpu().numpy(), ref)
        assert L.xamg_gs_plan_error(plan) == 0
    finally:
        L.xamg_gs_plan_destroy(plan)
