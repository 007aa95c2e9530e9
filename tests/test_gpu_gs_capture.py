"""A captured Gauss-Seidel call stays valid when the plan is used at a larger
width later, and the first call of a plan can be a captured one: the vector
between the two sweeps is never freed under a graph.  70^3 rows: the vector that
comes with the values holds 24 columns in FP64, so 32 need another.  Every sum
keeps its order, so replays are compared exactly."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import xamg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plan_of():
    d = sp.diags([-1.0, 2.0, -1.0], [-1, 0, 1], shape=(70, 70))
    e = sp.identity(70)
    A = (sp.kron(sp.kron(d, e), e) + sp.kron(sp.kron(e, d), e) + sp.kron(sp.kron(e, e), d)).tocsr()
    A.sort_indices()
    rp, ci, v = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    L = xamg.lib()
    made = []

    def make():
        p = L.xamg_gs_plan_create(A.shape[0], xamg._ptr(rp), xamg._ptr(ci), 0, 1)
        assert p
        made.append(p)
        xamg.check(L.xamg_gs_plan_set_values(p, xamg._ptr(v), 0))
        return p

    yield make, A.shape[0], (rp, ci, v)
    for p in made:
        L.xamg_gs_plan_destroy(p)


def vectors(n, arrays, nv):
    rng = np.random.default_rng(nv)
    h = [*arrays, np.full(n, 1.0 / 6.0), *(rng.uniform(-1, 1, (n, nv)) for _ in range(2)), np.full(nv, 0.99)]
    t = [torch.as_tensor(a).cuda() for a in h]
    torch.cuda.synchronize()
    return t


def call(plan, nv, t, stream=None):
    q = [a.data_ptr() for a in t]
    xamg.check(xamg.lib().xamg_hsgs(plan, 0, nv, q[0], q[1], q[2], q[3], q[4], q[5], q[6], None, stream))


def eager(plan, nv, n, arrays):
    t = vectors(n, arrays, nv)
    call(plan, nv, t)
    torch.cuda.synchronize()
    return t[5].cpu()


def captured(plan, nv, t):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(plan, nv, t, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return g


@pytest.mark.parametrize("first", [4, 32], ids=["within the vector", "first call, a wider vector"])
def test_replay(gpu, plan_of, first):
    make, n, arrays = plan_of
    ref = eager(make(), first, n, arrays)
    plan = make()
    t = vectors(n, arrays, first)
    x0 = t[5].clone()
    g = captured(plan, first, t)
    assert torch.equal(t[5], x0)  # captured, not run
    assert torch.equal(eager(plan, 32, n, arrays), eager(make(), 32, n, arrays))
    fill = [torch.full((n * 32,), 7.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    for _ in range(2):
        t[5].copy_(x0)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(t[5].cpu(), ref)
    assert all(bool((f == 7.0).all()) for f in fill)
    assert xamg.lib().xamg_gs_plan_error(plan) == 0
