"""One pair of FP32 vectors that do not both lie on a 16-byte boundary, and
operands beyond L2 whose chunks are split over warps: the sums keep their order,
so the oracle's values are matched exactly."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


def dot(prec, nv, n, pairs):
    L, nd = xamg.lib(), len(pairs)
    part = torch.empty(L.xamg_dot_part_size(n, nd, nv), dtype=torch.float64, device="cuda")
    out = torch.empty(nd * nv, dtype=torch.float64, device="cuda")
    a = (C.c_void_p * nd)(*[p.data_ptr() for p, _ in pairs])
    b = (C.c_void_p * nd)(*[p.data_ptr() for _, p in pairs])
    torch.cuda.synchronize()
    xamg.check(L.xamg_dot(prec, nv, n, nd, a, b, C.c_void_p(part.data_ptr()), C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("nv", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("shift", [(0, 2), (2, 0), (2, 2), (0, 0)])
@pytest.mark.parametrize("n", [300, 70001])
def test_eight_byte_boundaries(gpu, nv, shift, n):
    rng = np.random.default_rng(nv)
    h = [rng.uniform(-1, 1, (n, nv)).astype(np.float32) for _ in range(2)]
    d = []
    for a, k in zip(h, shift):
        t = torch.zeros(n * nv + 2, dtype=torch.float32, device="cuda")[k:k + n * nv]
        d.append(t.copy_(torch.as_tensor(a).reshape(-1)))
    np.testing.assert_array_equal(dot(1, nv, n, [(d[0], d[1])]), orc.dot(h[0], h[1]))


@pytest.mark.parametrize("dtype,nv,n", [(np.float64, 8, 900001), (np.float64, 4, 1800001), (np.float32, 32, 460001),
                                        (np.float32, 8, 1800001)])
def test_beyond_l2(gpu, dtype, nv, n):
    rng = np.random.default_rng(nv)
    h = [rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(2)]
    d = [torch.as_tensor(a).cuda() for a in h]
    prec = 0 if dtype == np.float64 else 1
    np.testing.assert_array_equal(dot(prec, nv, n, [(d[0], d[1])]), orc.dot(h[0], h[1]))
    ref = np.concatenate([orc.dot(h[0], h[1]), orc.dot(h[0], h[0]), orc.dot(h[1], h[1])])
    np.testing.assert_array_equal(dot(prec, nv, n, [(d[0], d[1]), (d[0], d[0]), (d[1], d[1])]), ref)
