"""The CSR product with a warp's rows side by side, and the default choice of
kernel for operators whose entries are counted: every row keeps its own chain
over its entries in stored order, so all kernels agree bit for bit with the
oracle.  Rows of 0, 1, a step (8, 16) and one more entry than a step, row
counts around a warp's and a block's rows, unsorted columns."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


def ragged(n, lengths, seed, dtype):
    rng = np.random.default_rng(seed)
    cnt = rng.choice(lengths, n)
    cnt[0] = max(lengths)
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    return rp, ci, rng.uniform(-1, 1, rp[-1]).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nv", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("n,lengths", [(1, [0, 5]), (7, [1, 8, 9]), (33, [0, 16, 17]), (128, [7, 24, 33]),
                                       (1027, [0, 3, 90]), (40001, [2, 40])])
def test_rows_side_by_side(gpu, dtype, nv, n, lengths):
    L = xamg.lib()
    rp, ci, v = ragged(n, lengths, n + nv, dtype)
    rng = np.random.default_rng(nv)
    x, y, b = (rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(3))
    d = [torch.as_tensor(a).cuda() for a in (rp, ci, v, x, b)]
    ptr = [C.c_void_p(t.data_ptr()) for t in d]
    prec = 0 if dtype == np.float64 else 1
    old = L.xamg_spmv_set_variant(-1)
    try:
        for variant in (8, -1):
            L.xamg_spmv_set_variant(variant)
            for mode in (0, 1, 2):
                out = torch.as_tensor(y).cuda()
                xamg.check(L.xamg_csr_spmv(prec, nv, n, ptr[0], ptr[1], ptr[2], ptr[3],
                                           C.c_void_p(out.data_ptr()), mode, ptr[4], None))
                torch.cuda.synchronize()
                ref = orc.spmv(rp, ci, v, x, nv, y=y.copy(), acc=True) if mode == 1 else orc.spmv(rp, ci, v, x, nv)
                if mode == 2:
                    ref = (dtype(1) * b + dtype(-1) * ref).astype(dtype)
                assert np.array_equal(out.cpu().numpy(), ref), (variant, mode)
    finally:
        L.xamg_spmv_set_variant(old)
