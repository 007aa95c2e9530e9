"""b - A x by the run product on either side of the line (80 MB of vectors and
values) from which b's lines are asked for ahead, in both kernel forms: the
oracle's values."""
import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,nv,n", [(np.float64, 16, 150000), (np.float64, 16, 200000), (np.float64, 32, 80000),
                                        (np.float64, 32, 100000), (np.float32, 32, 200000)])
@pytest.mark.parametrize("form", [0, 1])
def test_residual(gpu, dtype, nv, n, form):
    rng = np.random.default_rng(nv)
    r = np.arange(n)
    c = np.stack([r - 300, r - 1, r, r + 1, r + 300], 1)
    on = (c >= 0) & (c < n)
    on[::101, 3] = False  # chunks of every length, and rows by themselves
    rp = np.concatenate([[0], np.cumsum(on.sum(1))]).astype(np.int32)
    ci = c[on].astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1])
    L = xamg.lib()
    plan = L.xamg_spmv_runs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), xamg._ptr(v), 8, 0 if dtype == np.float64 else 1)
    assert plan
    old = L.xamg_spmv_set_run_form(form)
    try:
        x, b = (rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(2))
        d = [torch.as_tensor(a).cuda() for a in (x, b)]
        y = torch.zeros_like(d[0])
        torch.cuda.synchronize()
        xamg.check(L.xamg_spmv_runs(plan, 0 if dtype == np.float64 else 1, nv, d[0].data_ptr(), y.data_ptr(), 2,
                                    d[1].data_ptr(), None))
        torch.cuda.synchronize()
        ref = (dtype(1) * b + dtype(-1) * orc.spmv(rp, ci, v.astype(dtype), x, nv)).astype(dtype)
        assert np.array_equal(y.cpu().numpy(), ref)
    finally:
        L.xamg_spmv_set_run_form(old)
        L.xamg_spmv_runs_plan_destroy(plan)
