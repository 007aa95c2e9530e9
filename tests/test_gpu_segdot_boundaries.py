"""Per-segment inner products of vectors that start on any element: the loads
of two elements are used only where every vector lies on their boundary.  The
order of the sums does not depend on it: the oracle's values, exactly."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as orc
import xamg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nv", [1, 2, 4, 32])
@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (1, 1)])
def test_segments_from_any_element(gpu, dtype, nv, shift):
    L = xamg.lib()
    off = np.array([0, 3, 3, 260, 260 + 256, 1400], np.int64)
    n, nseg = int(off[-1]), len(off) - 1
    rng = np.random.default_rng(nv)
    h = [rng.uniform(-1, 1, (n, nv)).astype(dtype) for _ in range(2)]
    d = []
    for a, k in zip(h, shift):
        t = torch.zeros(n * nv + 1, dtype=torch.as_tensor(a).dtype, device="cuda")[k:k + n * nv]
        t.copy_(torch.as_tensor(a).reshape(-1))
        d.append(t)
    torch.cuda.synchronize()
    for pairs in ([(0, 1)], [(0, 1), (1, 1)], [(0, 1), (0, 0), (1, 1)], [(1, 0), (0, 0), (0, 1)]):
        nd = len(pairs)
        A = (C.c_void_p * nd)(*[d[i].data_ptr() for i, _ in pairs])
        B = (C.c_void_p * nd)(*[d[j].data_ptr() for _, j in pairs])
        out = torch.empty((nd, nseg, nv), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        xamg.check(L.xamg_seg_dot(0 if dtype == np.float64 else 1, nv, nseg, off.ctypes.data, nd, A, B,
                                  C.c_void_p(out.data_ptr()), None))
        got = out.cpu().numpy()
        for k, (i, j) in enumerate(pairs):
            for s in range(nseg):
                r = slice(int(off[s]), int(off[s + 1]))
                ref = orc.dot(h[i][r], h[j][r]) if off[s + 1] > off[s] else np.zeros(nv)
                np.testing.assert_array_equal(got[k, s], ref)
