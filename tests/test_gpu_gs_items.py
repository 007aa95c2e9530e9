"""Gauss-Seidel sweeps by items of one warp: rows longer than an item's staging
(over 256 entries), rows of a warp and of half a warp (NV 32), rows with only
their diagonal, a last block shorter than the others, and both sides of the
rule that runs a narrow schedule in one block.  Every row keeps the stored
order of its sum, so the oracle is matched exactly."""
import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


def system(n, width, long_rows, seed, gap=0):
    """Band of 2*width+1, `long_rows` rows coupled to 300 random others, every gap-th row diagonal only."""
    rng = np.random.default_rng(seed)
    extra = set(rng.choice(n, long_rows, replace=False).tolist()) if long_rows else set()
    rp, ci, v = [0], [], []
    for i in range(n):
        w = 0 if gap and i % gap == 0 else width
        c = set(range(max(0, i - w), min(n, i + w + 1)))
        if i in extra:
            c |= set(rng.choice(n, min(n, 300), replace=False).tolist())
        c = np.array(sorted(c))
        a = rng.uniform(-1, 1, len(c))
        a[c == i] = 1.0 + np.abs(a).sum()
        ci.append(c), v.append(a), rp.append(rp[-1] + len(c))
    return np.array(rp, np.int32), np.concatenate(ci).astype(np.int32), np.concatenate(v)


@pytest.mark.parametrize("n,width,long_rows,gap,brows", [
    (1, 0, 0, 0, 0), (130, 2, 0, 3, 0), (900, 1, 4, 0, 0),      # one item a level: one block
    (20000, 0, 3, 0, 0), (9000, 1, 2, 2, 0),                    # wide levels: the whole device
    (1300, 3, 2, 5, 500), (4097, 1, 3, 0, 64), (640, 9, 0, 0, 639),
])
@pytest.mark.parametrize("nv", [1, 2, 8, 32])
def test_items(gpu, n, width, long_rows, gap, brows, nv):
    rp, ci, v = system(n, width, long_rows, n + width, gap)
    L = xamg.lib()
    rng = np.random.default_rng(nv)
    plan = L.xamg_gs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), brows, 1)
    assert plan
    try:
        for dtype, prec in ((np.float64, 0), (np.float32, 1)):
            xamg.check(L.xamg_gs_plan_set_values(plan, xamg._ptr(v), prec))
            vv = v.astype(dtype)
            diag = np.array([vv[rp[i] + np.searchsorted(ci[rp[i]:rp[i + 1]], i)] for i in range(n)])
            invd = (1.0 / diag.astype(np.float64)).astype(dtype)
            b, x0 = (rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(2))
            relax = np.full(nv, 0.99, dtype)
            keep = [torch.as_tensor(a).cuda() for a in (rp, ci, vv, invd, b, x0, relax, np.zeros_like(b))]
            q = [t.data_ptr() for t in keep]
            xamg.check(L.xamg_hsgs(plan, prec, nv, q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], None))
            torch.cuda.synchronize()
            ref = orc.hsgs(rp, ci, vv, invd, b, x0.copy(), relax, block_rows=brows)
            assert np.array_equal(keep[5].cpu().numpy(), ref), dtype
        assert L.xamg_gs_plan_error(plan) == 0
    finally:
        L.xamg_gs_plan_destroy(plan)
