"""BiCGStab iterations in one launch: against the oracle, and against the
separate kernels (which the in-solve kernel timing selects), at the sizes where
the split into chunks of 256 rows, the copy of the matrix in shared memory and
the iterations per launch change.  All three run the same arithmetic in the
same order, so the comparison is exact."""
import numpy as np
import pytest

import oracle as orc
import util
import xamg

pytestmark = pytest.mark.gpu


def band(n, width, seed, gap=0):
    """Diagonally dominant rows of up to 2*width+1 random entries; every gap-th row only its diagonal."""
    rng = np.random.default_rng(seed)
    rp, ci, v = [0], [], []
    for i in range(n):
        w = 0 if gap and i % gap == 0 else width
        c = np.arange(max(0, i - w), min(n, i + w + 1))
        a = rng.uniform(-1, 1, len(c))
        a[c == i] = 1.0 + 1.1 * np.abs(a).sum()
        ci.append(c), v.append(a), rp.append(rp[-1] + len(c))
    return np.array(rp, np.int32), np.concatenate(ci).astype(np.int32), np.concatenate(v)


def laplace(n):
    rp, ci, v = [0], [], []
    for i in range(n):
        c = [j for j in (i - 1, i, i + 1) if 0 <= j < n]
        ci += c
        v += [2.0 if j == i else -1.0 for j in c]
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(v)


def run(arrays, B, iters, timed, meta=None):
    spec = util.amg_params(precond_mg=False, max_iters=iters, meta=meta)
    n, nv = B.shape
    xamg.set_nv(nv)
    A = xamg.Matrix(xamg.CsrMatrix.from_arrays(*arrays))
    x, b = xamg.Vector(n, nv), xamg.Vector(n, nv)
    x.upload(np.zeros_like(B))
    b.upload(B)
    s = xamg.Solver(A, xamg.Params(spec), x, b)
    xamg.kernel_timing(timed)
    try:
        s.solve()
    finally:
        xamg.kernel_timing(False)
    return x.download(), s.iters()[0], s.history()


CASES = [
    (1, 1, 0, 1, 50), (255, 3, 5, 1, 50), (256, 3, 0, 2, 50), (257, 2, 7, 4, 50), (1000, 3, 3, 8, 50),
    (513, 4, 0, 16, 50), (300, 2, 0, 32, 50),
    (700, 200, 0, 1, 50), (700, 200, 9, 8, 50),   # rows that do not fit in shared memory
    (148 * 256 + 1, 3, 11, 1, 50), (148 * 256 + 1, 3, 0, 8, 50),  # more than one chunk on an SM
    (2 * 148 * 256, 1, 0, 2, 20), (2 * 148 * 256 + 1, 1, 0, 2, 20),  # the largest, and one row more
    (1000, 3, 0, 4, 1), (1000, 3, 0, 1, 3),       # max_iters before convergence
]


@pytest.mark.parametrize("n,width,gap,nv,iters", CASES)
def test_iterations_match_oracle_and_separate_kernels(gpu, n, width, gap, nv, iters):
    arrays = band(n, width, 7 * n + nv, gap)
    B = np.random.default_rng(n + nv).uniform(-1, 1, (n, nv))
    x, it, hist = run(arrays, B, iters, False)
    x1, it1, hist1 = run(arrays, B, iters, True)
    xo, ito, histo, _, _ = orc.pbicgstab(*arrays, B, np.zeros_like(B), None, iters, 0.0, 1e-8)
    assert it == it1 == ito
    np.testing.assert_array_equal(hist, hist1)
    np.testing.assert_array_equal(x, x1)
    np.testing.assert_array_equal(hist, histo)
    np.testing.assert_array_equal(x, xo)


def test_iterations_continue_over_launches(gpu):
    # a launch holds 256 iterations; this system is far from converged after 600
    arrays = laplace(3000)
    B = np.random.default_rng(5).uniform(-1, 1, (3000, 2))
    x, it, hist = run(arrays, B, 600, False)
    x1, it1, hist1 = run(arrays, B, 600, True)
    assert it == it1 == 600
    np.testing.assert_array_equal(hist, hist1)
    np.testing.assert_array_equal(x, x1)


@pytest.mark.parametrize("nv", [1, 2, 4, 8, 16, 32])
def test_iterations_in_fp32(gpu, nv):
    # the inner solver of a refinement with reduced precision
    meta = {"method": "IterativeRefinement", "max_iters": 20, "abs_tolerance": 0.0, "rel_tolerance": 1e-9,
            "subsolver_reduced_precision": True, "inner_rel_tolerance": 1e-4,
            "convergence_details": "check-L2,noprint"}
    arrays = band(1500, 3, nv, 7)
    B = np.random.default_rng(nv).uniform(-1, 1, (1500, nv))
    x, it, hist = run(arrays, B, 60, False, meta)
    x1, it1, hist1 = run(arrays, B, 60, True, meta)
    assert it == it1 > 0
    np.testing.assert_array_equal(hist, hist1)
    np.testing.assert_array_equal(x, x1)
