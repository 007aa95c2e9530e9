"""Performance cases of the solve phase and of the learned initial guess.

Each case is one call (or one short sequence of calls) that a program makes
through the library's Python binding or its C entry points: whole solves
(plain, AMG-preconditioned, mixed precision, batched), the single kernels a
solver is composed of (products, Gauss-Seidel sweeps, inner products) and the
layers of the convolutional network (forward, backward).  `listed()` gives the
fixed cases, `draw()` one more of the same kinds with sizes spread over their
ranges, `exact()` the result in 64 bits by plain torch.

Operators are finite-volume stencils assembled here on the GPU: "poisson"
(7-point, unit coefficients), "lognormal" (7-point, lognormal cell
coefficients with harmonic face means) and "aniso" (27-point anisotropic
diffusion with axis coefficients 1, 1, 1e-3); "irregular" stands for a coarse
multigrid operator (rows of 8 to 120 entries scattered around the diagonal).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

os.environ.setdefault("XAMG_QUIET", "1")
sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "xamg-test_b200"))

DTYPE = {"f64": torch.float64, "f32": torch.float32}
PREC = {"f64": 0, "f32": 1}
BLOCKS = 444  # hybrid Gauss-Seidel blocks of the mixed form: three per SM


def listed():
    return [
        # the plain method's smallest configuration: 7-point Poisson, one
        # right-hand side, unpreconditioned BiCGStab
        dict(name="bicgstab_poisson32_nv1", kind="solve", form="bicgstab", op="poisson", nx=32, ny=32, nz=32, nv=1),
        # the FP64 drop-in: AMG-PBiCGStab, Gauss-Seidel in the single-process
        # row order, a few right-hand sides
        dict(name="amg_plain_aniso32_nv4", kind="solve", form="plain", op="aniso", nx=32, ny=32, nz=32, nv=4),
        # the precision form on many right-hand sides: FP64 refinement around
        # FP32 AMG-PBiCGStab with the hybrid smoother
        dict(name="amg_mixed_aniso64_nv16", kind="solve", form="mixed", op="aniso", nx=64, ny=64, nz=64, nv=16),
        # independent small systems of uneven size in one graph launch, with
        # the right-hand sides copied in and the solutions copied out
        dict(name="batch8_lognormal_16to40", kind="batch", systems=8, lo=16, hi=40),
        # one right-hand side, the commonest product, on a ragged grid
        dict(name="spmv_7pt_ragged_nv1_f64", kind="spmv", op="lognormal", nx=113, ny=97, nz=101, nv=1, dtype="f64",
             mode=0),
        # the finest operator's product of the 128^3 benchmark system
        dict(name="spmv_runs_aniso128_nv16_f64", kind="runs", op="aniso", nx=128, ny=128, nz=128, nv=16, dtype="f64",
             mode=0),
        # residual on a coarse level of an FP32 hierarchy
        dict(name="spmv_irregular56k_nv8_f32", kind="spmv", op="irregular", n=55799, nv=8, dtype="f32", mode=2),
        # the three fused inner products of one BiCGStab step
        dict(name="dots3_885k_nv16_f64", kind="dots", n=884736, nd=3, nv=16, dtype="f64"),
        # one symmetric Gauss-Seidel call, single-process row order, FP64
        dict(name="hsgs_sequential_aniso48_nv8_f64", kind="hsgs", op="aniso", nx=48, ny=48, nz=48, nv=8, dtype="f64",
             blocks=0),
        # one symmetric Gauss-Seidel call of the mixed form's smoother
        dict(name="hsgs_blocks_aniso80_nv16_f32", kind="hsgs", op="aniso", nx=80, ny=80, nz=80, nv=16, dtype="f32",
             blocks=BLOCKS),
        # the network's widest full-resolution layer, inference on 8 volumes
        dict(name="conv_48to16_64cube_x8", kind="conv", nb=8, d=64, h=64, w=64, cin=48, cout=16),
        # the backward of a decoder layer one level down: mask of the ReLU,
        # weight, bias and input gradients
        dict(name="conv_backward_96to32_32cube_x4", kind="conv_backward", nb=4, d=32, h=32, w=32, cin=96, cout=32),
    ]


LAYERS = [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (192, 64), (96, 32), (48, 16)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bicgstab", "plain", "mixed", "batch", "spmv", "irregular", "runs", "dots", "hsgs0", "hsgs",
                       "conv", "conv_backward"])
    if kind == "bicgstab":
        return dict(kind="solve", form="bicgstab", op=rng.choice(["poisson", "aniso"]), nx=rng.randint(10, 40),
                    ny=rng.randint(10, 40), nz=rng.randint(10, 40), nv=rng.choice([1, 1, 2, 4, 8, 16]))
    if kind == "plain":
        return dict(kind="solve", form="plain", op=rng.choice(["poisson", "aniso"]), nx=rng.randint(12, 32),
                    ny=rng.randint(12, 32), nz=rng.randint(12, 32), nv=rng.choice([1, 2, 4, 8]))
    if kind == "mixed":
        return dict(kind="solve", form="mixed", op="aniso", nx=rng.randint(24, 56), ny=rng.randint(24, 56),
                    nz=rng.randint(24, 56), nv=rng.choice([1, 4, 8, 16, 32]))
    if kind == "batch":
        lo = rng.randint(8, 20)
        return dict(kind="batch", systems=rng.randint(3, 9), lo=lo, hi=rng.randint(lo + 4, 36))
    if kind == "spmv":
        return dict(kind="spmv", op=rng.choice(["poisson", "lognormal", "aniso"]), nx=_log(rng, 12, 100),
                    ny=_log(rng, 12, 100), nz=_log(rng, 12, 100), nv=rng.choice([1, 2, 4, 8, 16, 32]),
                    dtype=rng.choice(["f64", "f32"]), mode=rng.choice([0, 1, 2]))
    if kind == "irregular":
        return dict(kind="spmv", op="irregular", n=_log(rng, 300, 80000), nv=rng.choice([1, 2, 4, 8, 16]),
                    dtype=rng.choice(["f64", "f32"]), mode=rng.choice([0, 1, 2]))
    if kind == "runs":
        dtype, nv = rng.choice([("f64", 8), ("f64", 16), ("f64", 32), ("f32", 16), ("f32", 32)])
        return dict(kind="runs", op=rng.choice(["lognormal", "aniso"]), nx=rng.randint(20, 90), ny=rng.randint(20, 90),
                    nz=rng.randint(20, 90), nv=nv, dtype=dtype, mode=rng.choice([0, 1, 2]))
    if kind == "dots":
        nv = rng.choice([1, 2, 4, 8, 16, 32])
        return dict(kind="dots", n=_log(rng, 1000, 8000000 // nv), nd=rng.randint(1, 4), nv=nv,
                    dtype=rng.choice(["f64", "f32"]))
    if kind in ("hsgs0", "hsgs"):
        return dict(kind="hsgs", op=rng.choice(["lognormal", "aniso"]), nx=rng.randint(12, 56), ny=rng.randint(12, 56),
                    nz=rng.randint(12, 56), nv=rng.choice([1, 2, 4, 8, 16, 32]), dtype=rng.choice(["f64", "f32"]),
                    blocks=0 if kind == "hsgs0" else rng.choice([16, 148, 296, BLOCKS]))
    cin, cout = rng.choice(LAYERS)
    side = rng.choice([3, 6, 8, 12, 16, 20, 24, 32, 40]) if cin <= 96 else rng.choice([3, 5, 8, 10, 16, 20])
    most = 8 if kind == "conv" else max(1, min(8, 12000000 // (cin * side ** 3)))
    return dict(kind=kind, nb=rng.randint(1, most), d=side, h=side, w=side, cin=cin, cout=cout)


# ------------------------------------------------------------------ operators
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") * 2.0 - 1.0


def _stencil(c, seed):
    """(columns [n, k] int32, values [n, k] FP64, present [n, k]) of a stencil
    operator, the diagonal first and then the neighbours in (z, y, x) order."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    n = nx * ny * nz
    r = torch.arange(n, device="cuda", dtype=torch.int32)
    i, j, k = r % nx, (r // nx) % ny, r // (nx * ny)
    wide = c["op"] == "aniso"
    offs = [(a, b, e) for a in (-1, 0, 1) for b in (-1, 0, 1) for e in (-1, 0, 1)
            if (a, b, e) != (0, 0, 0) and (wide or abs(a) + abs(b) + abs(e) == 1)]
    cols = torch.zeros((n, len(offs) + 1), dtype=torch.int32, device="cuda")
    vals = torch.zeros((n, len(offs) + 1), dtype=torch.float64, device="cuda")
    on = torch.ones((n, len(offs) + 1), dtype=torch.bool, device="cuda")
    cols[:, 0] = r
    cell = torch.exp(torch.randn((n,), generator=_gen(seed + 7), dtype=torch.float64, device="cuda")) \
        if c["op"] == "lognormal" else None
    for q, (dz, dy, dx) in enumerate(offs):
        ii, jj, kk = i + dx, j + dy, k + dz
        ok = (ii >= 0) & (ii < nx) & (jj >= 0) & (jj < ny) & (kk >= 0) & (kk < nz)
        col = torch.where(ok, (kk * ny + jj) * nx + ii, 0)
        if wide:
            d2 = dx * dx + dy * dy + dz * dz
            w = torch.full((n,), (dx * dx + dy * dy + 1e-3 * dz * dz) / float(d2 * d2), dtype=torch.float64,
                           device="cuda")
        elif cell is None:
            w = torch.ones((n,), dtype=torch.float64, device="cuda")
        else:  # harmonic mean of the two cells, the cell itself on the boundary
            o = cell[col.long()]
            w = torch.where(ok, 2.0 * cell * o / (cell + o), cell)
        vals[:, 0] += w
        cols[:, q + 1], vals[:, q + 1], on[:, q + 1] = col, torch.where(ok, -w, 0.0), ok
    return cols, vals, on


def _irregular(c, seed):
    """Rows of 8 to 120 entries (log-uniform) around the diagonal, the
    diagonal first and dominant."""
    n, g = c["n"], _gen(seed + 7)
    u = torch.rand((n,), generator=g, device="cuda", dtype=torch.float64)
    cnt = torch.exp(math.log(8.0) + u * math.log(120.0 / 8.0)).to(torch.int64).clamp(max=n)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(cnt, 0)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), cnt)
    nnz = row.numel()
    off = torch.randn((nnz,), generator=g, device="cuda", dtype=torch.float64) * min(2000.0, n / 4.0)
    ci = (row + off.to(torch.int64)).clamp(0, n - 1)
    v = -torch.rand((nnz,), generator=g, device="cuda", dtype=torch.float64)
    ci[rp[:-1]], v[rp[:-1]] = torch.arange(n, device="cuda"), cnt.to(torch.float64)
    return rp.to(torch.int32), ci.to(torch.int32), v


def _csr(c, seed):
    """Device CSR arrays (int32, int32, FP64) of the case's operator."""
    if c["op"] == "irregular":
        return _irregular(c, seed)
    cols, vals, on = _stencil(c, seed)
    rp = torch.zeros(cols.shape[0] + 1, dtype=torch.int32, device="cuda")
    rp[1:] = torch.cumsum(on.sum(1), 0)
    return rp, cols[on], vals[on]


def _rows(c):
    return c["n"] if "n" in c else c["nx"] * c["ny"] * c["nz"]


def _nnz(c):
    if c["op"] == "irregular":
        return _rows(c) * 41.4  # mean of the log-uniform row lengths
    x, y, z = c["nx"], c["ny"], c["nz"]
    if c["op"] == "aniso":
        return (3 * x - 2) * (3 * y - 2) * (3 * z - 2)
    return 7 * x * y * z - 2 * (x * y + y * z + x * z)


def _host(*t):
    return [a.cpu().numpy() for a in t]


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _batch_members(c, seed):
    """[(side, nv)] of the batch: sides log-uniform, widths 1, 2, 4 and 8.
    The shapes belong to the case, the coefficients and right-hand sides to
    the seed."""
    rng = np.random.default_rng(c["systems"] * 1000 + c["lo"] * 50 + c["hi"])
    sides = [int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]))))) for _ in range(c["systems"])]
    return [(s, int(rng.choice([1, 2, 4, 8]))) for s in sides]


# ---------------------------------------------------------------- inputs
def _vectors(c, seed):
    """b, x0 of a solve or sweep, or x, y, b of a product, uniform in [-1, 1]."""
    g = _gen(seed)
    n, nv = _rows(c), c["nv"]
    dt = DTYPE[c.get("dtype", "f64")]
    return [_uniform(g, n, nv).to(dt) for _ in range(3)]


def _dot_vectors(c, seed):
    g = _gen(seed)
    dt = DTYPE[c["dtype"]]
    return [_uniform(g, c["n"], c["nv"]).to(dt) for _ in range(2 * c["nd"])]


def _conv_inputs(c, seed):
    """Input activations (after a ReLU: half of them zero), weights (He
    scaling), biases, the layer's output and the gradient that reaches it."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = (c["nb"], c["d"], c["h"], c["w"])
    bf = torch.bfloat16

    def rnd(*s):
        return torch.randn(s, generator=g, device="cuda")

    x = torch.relu(rnd(*shape, c["cin"])).to(bf)
    w = (rnd(c["cout"], 27, c["cin"]) * (2.0 / (27 * c["cin"])) ** 0.5).to(bf)
    bias = 0.1 * rnd(c["cout"])
    act = torch.relu(rnd(*shape, c["cout"])).to(bf)
    grad = rnd(*shape, c["cout"]).to(bf)
    return x, w, bias, act, grad


# ------------------------------------------------------------------- solves
def _spec(form):
    spec = {"solver": {"method": "BiCGStab" if form == "bicgstab" else "PBiCGStab", "max_iters": 400,
                       "abs_tolerance": 0.0, "rel_tolerance": 1e-8, "convergence_details": "check-L2,noprint"}}
    if form == "bicgstab":
        return spec
    hybrid = {"hybrid_blocks": BLOCKS} if form == "mixed" else {}
    spec["preconditioner"] = {"method": "MultiGrid", "mg_coarsening_type": 10, "mg_interpolation_type": 6,
                              "mg_strength_threshold": 0.25, "mg_max_levels": 6, "mg_agg_num_levels": 0}
    spec["pre_smoother"] = dict({"method": "HSGS", "max_iters": 1}, **hybrid)
    spec["post_smoother"] = dict({"method": "HSGS", "max_iters": 1}, **hybrid)
    spec["coarse_grid_solver"] = {"method": "Direct"}
    if form == "mixed":
        spec["meta_solver"] = {"method": "IterativeRefinement", "max_iters": 20, "abs_tolerance": 0.0,
                               "rel_tolerance": 1e-8, "subsolver_reduced_precision": True,
                               "inner_rel_tolerance": 1e-4, "convergence_details": "check-L2,noprint"}
    return spec


class _DeviceVector:
    """A library vector as a torch tensor without a copy; keeps its owners."""

    def __init__(self, vec, *owners):
        self.owners = (vec,) + owners
        self.__cuda_array_interface__ = {"shape": (vec.n, vec.nv), "typestr": "<f8", "version": 3, "strides": None,
                                         "data": (int(vec.device_ptr), False)}


class _Plan:
    """A plan handle of the C interface, destroyed with this object."""

    def __init__(self, handle, destroy):
        import xamg
        if not handle:
            raise RuntimeError(xamg.lib().XAMG_b200_last_error().decode())
        self.h, self.destroy = handle, destroy

    def __del__(self):
        self.destroy(self.h)


def prepare(case, seed):
    import xamg
    c, kind = case, case["kind"]
    L = xamg.lib()
    s = {"case": c, "xamg": xamg, "L": L}
    if kind == "solve":
        xamg.init(c["nv"])
        csr = xamg.CsrMatrix.from_arrays(*_host(*_csr(c, seed)))
        A = xamg.Matrix(csr)
        x, b = xamg.Vector(csr.nrows, c["nv"]), xamg.Vector(csr.nrows, c["nv"])
        b.upload(_vectors(c, seed)[0].cpu().numpy())
        s.update(x=x, solver=xamg.Solver(A, xamg.Params(_spec(c["form"])), x, b))
        s["view"] = torch.as_tensor(_DeviceVector(x, s["solver"]), device="cuda")
    elif kind == "batch":
        import families
        xamg.init(1)
        systems, rhs = [], []
        for q, (side, nv) in enumerate(_batch_members(c, seed)):
            m = dict(op="lognormal", nx=side, ny=side, nz=side, nv=nv)
            systems.append((xamg.CsrMatrix.from_arrays(*_host(*_csr(m, seed + 100 * q))), nv))
            rhs.append(_vectors(m, seed + 100 * q)[0].cpu().numpy())
        s.update(batch=xamg.Batch(systems, xamg.Params(families.batch_spec())), rhs=rhs)
    elif kind == "spmv":
        rp, ci, v = _csr(c, seed)
        x, y, b = _vectors(c, seed)
        s.update(rp=rp, ci=ci, v=v.to(DTYPE[c["dtype"]]), x=x, y=y, y0=y.clone(), b=b)
    elif kind == "runs":
        rp, ci, v = _host(*_csr(c, seed))
        x, y, b = _vectors(c, seed)
        plan = L.xamg_spmv_runs_plan_create(_rows(c), xamg._ptr(rp), xamg._ptr(ci), xamg._ptr(v), 8,
                                            PREC[c["dtype"]])
        s.update(plan=_Plan(plan, L.xamg_spmv_runs_plan_destroy), x=x, y=y, y0=y.clone(), b=b)
    elif kind == "dots":
        v = _dot_vectors(c, seed)
        nd = c["nd"]
        part = torch.empty(L.xamg_dot_part_size(c["n"], nd, c["nv"]), dtype=torch.float64, device="cuda")
        s.update(v=v, part=part, out=torch.empty((nd, c["nv"]), dtype=torch.float64, device="cuda"),
                 a=(C.c_void_p * nd)(*[t.data_ptr() for t in v[:nd]]),
                 b=(C.c_void_p * nd)(*[t.data_ptr() for t in v[nd:]]))
    elif kind == "hsgs":
        drp, dci, dv = _csr(c, seed)
        rp, ci, v = _host(drp, dci, dv)
        n, dt = _rows(c), DTYPE[c["dtype"]]
        rows = -(-n // c["blocks"]) if c["blocks"] else 0
        plan = _Plan(L.xamg_gs_plan_create(n, xamg._ptr(rp), xamg._ptr(ci), rows, 1), L.xamg_gs_plan_destroy)
        xamg.check(L.xamg_gs_plan_set_values(plan.h, xamg._ptr(v), PREC[c["dtype"]]))
        b, x, t = _vectors(c, seed)
        invd = 1.0 / dv[drp[:-1].long()].to(dt).to(torch.float64)
        s.update(plan=plan, rp=drp, ci=dci, v=dv.to(dt), b=b, x=x, t=t, invd=invd.to(dt),
                 relax=torch.ones(c["nv"], dtype=dt, device="cuda"))
    else:
        import learned
        s["L"] = learned.klib()
        x, w, bias, act, grad = _conv_inputs(c, seed)
        s.update(x=x, w=w, bias=bias, act=act, grad=grad, wt=torch.empty((c["cin"], 27, c["cout"]),
                                                                        dtype=torch.bfloat16, device="cuda"))
        s["y"] = torch.empty_like(act)
        if kind == "conv_backward":
            s.update(gw=torch.zeros((c["cout"], 27, c["cin"]), device="cuda"),
                     gb=torch.zeros(c["cout"], device="cuda"), gin=torch.empty_like(x))
    return s


def run(s):
    c, L, ok = s["case"], s["L"], s["xamg"].check
    kind = c["kind"]
    if kind == "solve":
        s["xamg"].set_nv(c["nv"])
        s["x"].set(0.0)
        s["solver"].solve()
        its = s["solver"].iters()
        return {"x": s["view"], "iterations": its[0], "inner": its[1]}
    if kind == "batch":
        for q, b in enumerate(s["rhs"]):
            s["batch"].upload(q, b)
        s["batch"].solve()
        return [s["batch"].download(q) for q in range(len(s["rhs"]))]
    if kind == "spmv":
        if c["mode"] == 1:  # the accumulating product starts from the same y in every pass
            s["y"].copy_(s["y0"])
            torch.cuda.current_stream().synchronize()
        ok(L.xamg_csr_spmv(PREC[c["dtype"]], c["nv"], _rows(c), _ptr(s["rp"]), _ptr(s["ci"]), _ptr(s["v"]),
                           _ptr(s["x"]), _ptr(s["y"]), c["mode"], _ptr(s["b"]), None))
        return s["y"]
    if kind == "runs":
        if c["mode"] == 1:
            s["y"].copy_(s["y0"])
            torch.cuda.current_stream().synchronize()
        ok(L.xamg_spmv_runs(s["plan"].h, PREC[c["dtype"]], c["nv"], _ptr(s["x"]), _ptr(s["y"]), c["mode"],
                            _ptr(s["b"]), None))
        return s["y"]
    if kind == "dots":
        ok(L.xamg_dot(PREC[c["dtype"]], c["nv"], c["n"], c["nd"], s["a"], s["b"], _ptr(s["part"]), _ptr(s["out"]),
                      None))
        return s["out"]
    if kind == "hsgs":  # one more smoothing step on the state's x
        ok(L.xamg_hsgs(s["plan"].h, PREC[c["dtype"]], c["nv"], _ptr(s["rp"]), _ptr(s["ci"]), _ptr(s["v"]),
                       _ptr(s["invd"]), _ptr(s["b"]), _ptr(s["x"]), _ptr(s["relax"]), _ptr(s["t"]), None))
        return s["x"]
    ci, co, vol = c["cin"], c["cout"], (c["nb"], c["d"], c["h"], c["w"])
    if kind == "conv":
        ok(L.xcnn_conv3d(_ptr(s["x"]), ci, 0, ci, _ptr(s["w"]), _ptr(s["bias"]), _ptr(s["y"]), co, 0, co, *vol, 1,
                         None))
        return s["y"]
    nvox = vol[0] * vol[1] * vol[2] * vol[3]
    s["gw"].zero_()
    s["gb"].zero_()
    ok(L.xcnn_relu_bwd(_ptr(s["grad"]), co, 0, _ptr(s["act"]), co, 0, co, nvox, None))
    ok(L.xcnn_conv3d_wgrad(_ptr(s["x"]), ci, 0, ci, _ptr(s["grad"]), co, 0, co, _ptr(s["gw"]), *vol, None))
    ok(L.xcnn_bias_grad(_ptr(s["grad"]), co, 0, co, nvox, _ptr(s["gb"]), None))
    ok(L.xcnn_weight_flip(_ptr(s["w"]), _ptr(s["wt"]), co, ci, None))
    ok(L.xcnn_conv3d(_ptr(s["grad"]), co, 0, co, _ptr(s["wt"]), None, _ptr(s["gin"]), ci, 0, ci, *vol, 0, None))
    return {"gw": s["gw"], "gb": s["gb"], "gin": s["gin"], "grad": s["grad"]}


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        n = sum(s ** 3 * (13 * 12 + 8 * 16 * v) for s, v in _batch_members(c, 0))
        return {"bytes": 8.0 * n, "flops": 8.0 * sum(s ** 3 * 60 * v for s, v in _batch_members(c, 0))}
    if kind == "dots":
        e = c["n"] * c["nv"] * c["nd"]
        return {"bytes": 2.0 * e * (8 if c["dtype"] == "f64" else 4), "flops": 2.0 * e}
    if kind in ("conv", "conv_backward"):
        vox = c["nb"] * c["d"] * c["h"] * c["w"]
        macs = 27.0 * vox * c["cin"] * c["cout"]
        if kind == "conv":
            return {"bytes": 2.0 * vox * (c["cin"] + c["cout"]) + 54.0 * c["cin"] * c["cout"], "flops": 2.0 * macs}
        return {"bytes": 2.0 * vox * (2 * c["cin"] + 3 * c["cout"]) + 162.0 * c["cin"] * c["cout"],
                "flops": 4.0 * macs}
    n, nnz, nv = _rows(c), _nnz(c), c["nv"]
    if kind == "solve":
        # nominal iteration counts of the forms; an iteration takes two
        # products of the operator (and, preconditioned, two V-cycles of about
        # six operator passes each on a hierarchy of complexity 1.7)
        its, passes = {"bicgstab": (2.6 * max(c["nx"], c["ny"], c["nz"]), 2), "plain": (4, 2 + 2 * 6 * 1.7),
                       "mixed": (5, 2 + 2 * 6 * 1.7)}[c["form"]]
        sv = 4 if c["form"] == "mixed" else 8
        per = nnz * (sv + 4) + 4.0 * n * nv * sv
        return {"bytes": its * passes * per, "flops": its * passes * 2.0 * nnz * nv}
    sv = 8 if c["dtype"] == "f64" else 4
    if kind == "hsgs":  # two sweeps over the operator
        return {"bytes": 2.0 * nnz * (sv + 4) + n * (4.0 + sv) + 3.0 * n * nv * sv, "flops": 4.0 * nnz * nv}
    return {"bytes": nnz * (sv + 4.0) + 4.0 * n + n * nv * sv * (2.0 + (c["mode"] > 0)), "flops": 2.0 * nnz * nv}


# ------------------------------------------------------------- 64-bit results
def _spd_solve(rp, ci, v, b):
    """Conjugate gradients with Jacobi scaling to 1e-13, in 64 bits."""
    n = rp.numel() - 1
    A = torch.sparse_csr_tensor(rp, ci, v, size=(n, n))
    di = (1.0 / v[rp[:-1].long()]).unsqueeze(1)
    x = torch.zeros_like(b)
    r = b.clone()
    z = di * r
    p = z.clone()
    rz = (r * z).sum(0)
    stop = 1e-13 * torch.linalg.vector_norm(b, dim=0)
    for it in range(4000):
        q = A @ p
        alpha = rz / (p * q).sum(0)
        x += alpha * p
        r -= alpha * q
        if it % 25 == 24 and bool((torch.linalg.vector_norm(r, dim=0) <= stop).all()):
            break
        z = di * r
        new = (r * z).sum(0)
        p = z + (new / rz) * p
        rz = new
    return x


def _sgs(c, seed):
    """One symmetric Gauss-Seidel step by wavefronts of independent rows."""
    cols, vals, on = _stencil(c, seed)
    vals = vals.to(DTYPE[c["dtype"]]).to(torch.float64)
    cols = cols.long()
    n = cols.shape[0]
    b, x, _ = [t.to(torch.float64) for t in _vectors(c, seed)]
    invd = (1.0 / vals[:, 0]).unsqueeze(1)
    r = torch.arange(n, device="cuda")
    t = b
    if c["blocks"]:
        rows = -(-n // c["blocks"])
        off = on & ((cols // rows) != (r // rows).unsqueeze(1))
        t = b.clone()
        for q in range(cols.shape[1]):
            t -= (vals[:, q] * off[:, q]).unsqueeze(1) * x[cols[:, q]]
        vals = torch.where(off, 0.0, vals)
    lev = r % c["nx"] + 2 * ((r // c["nx"]) % c["ny"]) + 4 * (r // (c["nx"] * c["ny"]))
    order = torch.argsort(lev, stable=True)
    ends = torch.cumsum(torch.bincount(lev), 0).tolist()
    groups = [order[a:z] for a, z in zip([0] + ends[:-1], ends)]
    for sweep in (groups, groups[::-1]):
        for g in sweep:
            s = t[g] - (vals[g].unsqueeze(2) * x[cols[g]]).sum(1)
            x[g] += invd[g] * s
    return x


def _shifted(x, t):
    """x [nb, d, h, w, c] at the voxels' neighbours of tap t, zero outside."""
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    z, y, w = t // 9, (t // 3) % 3, t % 3
    return p[:, z:z + x.shape[1], y:y + x.shape[2], w:w + x.shape[3]]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        x = _spd_solve(*_csr(c, seed), _vectors(c, seed)[0])
        return {"x": x, "iterations": None, "inner": None}
    if kind == "batch":
        out = []
        for q, (side, nv) in enumerate(_batch_members(c, seed)):
            m = dict(op="lognormal", nx=side, ny=side, nz=side, nv=nv)
            out.append(_spd_solve(*_csr(m, seed + 100 * q), _vectors(m, seed + 100 * q)[0]))
        return out
    if kind in ("spmv", "runs"):
        rp, ci, v = _csr(c, seed)
        v = v.to(DTYPE[c["dtype"]]).to(torch.float64)
        x, y, b = [t.to(torch.float64) for t in _vectors(c, seed)]
        n = rp.numel() - 1
        p = torch.sparse_csr_tensor(rp, ci, v, size=(n, n)) @ x
        return p if c["mode"] == 0 else y + p if c["mode"] == 1 else b - p
    if kind == "dots":
        v = _dot_vectors(c, seed)
        nd = c["nd"]
        return torch.stack([(v[d].to(torch.float64) * v[nd + d].to(torch.float64)).sum(0) for d in range(nd)])
    if kind == "hsgs":
        return _sgs(c, seed)
    x, w, bias, act, grad = _conv_inputs(c, seed)
    x, w = x.to(torch.float64), w.to(torch.float64)
    if kind == "conv":
        y = bias.to(torch.float64).expand(*act.shape).contiguous()
        for t in range(27):
            y += _shifted(x, t) @ w[:, t].T
        return torch.relu(y)
    g = torch.where(act > 0, grad, 0).to(torch.float64)
    flat = g.reshape(-1, c["cout"])
    gw = torch.stack([flat.T @ _shifted(x, t).reshape(-1, c["cin"]) for t in range(27)], 1)
    gin = torch.zeros_like(x)
    for t in range(27):
        gin += _shifted(g, 26 - t) @ w[:, t]
    return {"gw": gw, "gb": flat.sum(0), "gin": gin, "grad": g}
