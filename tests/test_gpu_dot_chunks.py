"""Inner products at the edges of their split: chunks of 256 rows, one or
several warps to a chunk, one warp or eight to a block, the pairs (a, b),
(a, a), (b, b) read once.  The order of the sums is fixed, so the oracle's
values are matched exactly."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nv", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 2049, 256 * 296 + 5, 256 * 2368 - 1])
def test_dots(gpu, dtype, nv, n):
    if n * nv > 256 * 2368 * 4:
        n //= 8  # the same split at a lower count of chunks
    L = xamg.lib()
    rng = np.random.default_rng(n + nv)
    h = [rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(4)]
    d = [torch.as_tensor(a).cuda() for a in h]
    part = torch.empty(L.xamg_dot_part_size(n, 4, nv), dtype=torch.float64, device="cuda")
    for pairs in ([(0, 1)], [(0, 1), (2, 3)], [(0, 1), (0, 0), (1, 1)], [(0, 1), (1, 2), (2, 0)],
                  [(0, 1), (1, 2), (2, 3), (3, 3)]):
        nd = len(pairs)
        out = torch.empty(nd * nv, dtype=torch.float64, device="cuda")
        a = (C.c_void_p * nd)(*[d[i].data_ptr() for i, _ in pairs])
        b = (C.c_void_p * nd)(*[d[j].data_ptr() for _, j in pairs])
        xamg.check(L.xamg_dot(0 if dtype == np.float64 else 1, nv, n, nd, a, b, C.c_void_p(part.data_ptr()),
                               C.c_void_p(out.data_ptr()), None))
        torch.cuda.synchronize()
        ref = np.concatenate([orc.dot(h[i], h[j]) for i, j in pairs])
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
