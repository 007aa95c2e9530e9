"""Which systems run whole BiCGStab iterations in one launch: those whose matrix
rows fit in the blocks' shared memory, decided by every block's own entries.
Counted by the launches of a solve; the results are the oracle's either way."""
import numpy as np
import pytest

import oracle as orc
import util
import xamg

pytestmark = pytest.mark.gpu


def system(n, width, dense_rows, seed):
    """Band of 2*width+1; the last dense_rows rows have 400 entries."""
    rng = np.random.default_rng(seed)
    rp, ci, v = [0], [], []
    for i in range(n):
        c = np.arange(max(0, i - width), min(n, i + width + 1))
        if i >= n - dense_rows:
            c = np.unique(np.concatenate([c, rng.choice(n, 400, replace=False)]))
        a = rng.uniform(-1, 1, len(c))
        a[c == i] = 1.0 + 1.1 * np.abs(a).sum()
        ci.append(c), v.append(a), rp.append(rp[-1] + len(c))
    return np.array(rp, np.int32), np.concatenate(ci).astype(np.int32), np.concatenate(v)


@pytest.mark.parametrize("n,width,dense,nv,one", [
    (2000, 3, 0, 1, True), (2000, 30, 0, 8, True), (2000, 30, 0, 16, False),  # 61 entries a row
    (2000, 45, 0, 1, False),
    (2000, 3, 20, 1, True), (2000, 3, 200, 1, False),  # one block with many entries
    (148 * 256 + 300, 14, 0, 1, True), (148 * 256 + 300, 18, 0, 1, False),  # two blocks on an SM
])
def test_choice(gpu, n, width, dense, nv, one):
    arrays = system(n, width, dense, n + width)
    B = np.random.default_rng(nv).uniform(-1, 1, (n, nv))
    xamg.set_nv(nv)
    A = xamg.Matrix(xamg.CsrMatrix.from_arrays(*arrays))
    x, b = xamg.Vector(n, nv), xamg.Vector(n, nv)
    x.upload(np.zeros_like(B))
    b.upload(B)
    s = xamg.Solver(A, xamg.Params(util.amg_params(precond_mg=False, max_iters=12)), x, b)
    before = xamg.kernel_launches()
    s.solve()
    it, count = s.iters()[0], xamg.kernel_launches() - before
    assert it >= 4 and (count < 10) == one, (it, count)
    xo, ito, histo, _, _ = orc.pbicgstab(*arrays, B, np.zeros_like(B), None, 12, 0.0, 1e-8)
    assert it == ito
    np.testing.assert_array_equal(s.history(), histo)
    np.testing.assert_array_equal(x.download(), xo)
