"""The work that programs give this library, as cases for timing: matrix products and
hand-written iterations, assembly and Galerkin products, and whole solves (CG, BiCGStab, GMRES,
multigrid-preconditioned CG, batches, a differentiable solve), each through the public entry
points (faspxx_b200.sol, faspxx_b200.autograd and the C ABI of include/fasp_b200.h).

Vectors live in torch tensors on the GPU. The C ABI's stream-ordered calls take torch's current
stream, so a solve starts after the torch work that forms its inputs.
"""
import ctypes as C
import math

import numpy as np
import torch

from faspxx_b200 import capi, sol
from faspxx_b200.autograd import SparseSystem, sparse_solve
from faspxx_b200.capi import check, lib

F64 = torch.float64


# ---- the cases -------------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: one step of a CG written by hand on MAT and VEC, on a small 2D grid
        {"name": "step_2d_65", "family": "step", "m": 65},
        # operator application, residual and transposed product on a large matrix with a
        # coefficient per cell (plain CSR, seven entries a row): what an outer solver, an
        # eigenvalue iteration or an explicit time step asks of MAT
        {"name": "product_var_160", "family": "product", "kind": "var", "m": 160},
        # the same on a finite-element matrix: up to 27 entries a row, ragged rows, nodes
        # numbered irregularly
        {"name": "product_fem_83", "family": "product", "kind": "fem", "m": 83},
        # the library's headline: Jacobi-PCG on the 3D Poisson matrix to 1e-8, in FP64 ...
        {"name": "cg_poisson_128", "family": "cg", "dim": 3, "m": 128, "precision": "fp64"},
        # ... and with FP32 iterations inside FP64 reliable updates
        {"name": "cg_mixed_128", "family": "cg", "dim": 3, "m": 128, "precision": "mixed"},
        # an implicit time step of convection-diffusion (a few BiCGStab iterations), odd size
        {"name": "bicgstab_101", "family": "bicgstab", "m": 101, "peclet": 0.5, "step": 1.0},
        # steady convection-diffusion with GMRES(30)
        {"name": "gmres_96", "family": "gmres", "m": 96, "peclet": 0.1},
        # multigrid V(2,2) as the preconditioner of CG
        {"name": "mgcg_127", "family": "mgcg", "m": 127},
        # a multigrid level for new coefficients: restriction, A P and R (A P)
        {"name": "galerkin_63", "family": "galerkin", "m": 63},
        # a matrix from shuffled triplets (a finite-element assembly or a .mtx file), applied once
        {"name": "assemble_64", "family": "assemble", "m": 64},
        # a training step: coefficients in, solution and gradients of coefficients and right-hand
        # side out
        {"name": "train_64", "family": "train", "m": 64},
        # many small uneven systems at once, four right-hand sides each
        {"name": "batch_512", "family": "batch", "count": 512, "lo": 16, "hi": 128, "nrhs": 4,
         "precision": "fp64"},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    f = rng.choice(["step", "product", "product", "cg", "cg", "bicgstab", "gmres", "mgcg",
                    "galerkin", "assemble", "train", "batch"])
    if f == "step":
        return {"family": f, "m": _spread(rng, 20, 400)}
    if f == "product":
        kind = rng.choice(["var", "fem", "poisson"])
        return {"family": f, "kind": kind, "m": _spread(rng, 12, 83 if kind == "fem" else 160)}
    if f == "cg":
        dim = rng.choice([2, 3, 3])
        return {"family": f, "dim": dim, "m": _spread(rng, 40, 400) if dim == 2 else
                _spread(rng, 20, 128), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if f == "bicgstab":
        return {"family": f, "m": _spread(rng, 16, 112), "peclet": round(rng.uniform(0.1, 2.0), 3),
                "step": round(rng.uniform(0.25, 1.5), 3)}
    if f == "gmres":
        return {"family": f, "m": _spread(rng, 16, 96), "peclet": round(rng.uniform(0.1, 2.0), 3)}
    if f == "mgcg":
        return {"family": f, "m": rng.choice([15, 23, 31, 39, 47, 55, 63, 79, 95, 111, 127])}
    if f == "galerkin":
        return {"family": f, "m": 2 * _spread(rng, 6, 31) + 1}
    if f == "assemble":
        return {"family": f, "m": _spread(rng, 8, 64)}
    if f == "train":
        return {"family": f, "m": _spread(rng, 12, 64)}
    lo = rng.randint(8, 32)
    return {"family": f, "count": _spread(rng, 24, 512), "lo": lo, "hi": rng.randint(lo + 16, 128),
            "nrhs": rng.randint(1, 4), "precision": rng.choice(["fp64", "fp64", "mixed"])}


# ---- inputs ----------------------------------------------------------------------------

class _Vec(sol.DVec):
    """A torch tensor where MAT's members take a DVec."""

    def __init__(self, t):
        self.t, self.n, self.ptr = t, t.numel(), C.c_void_p(t.data_ptr())

    def __del__(self):
        pass


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda", dtype=F64) * (hi - lo) + lo


_OFF2 = [(0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0)]
_OFF3 = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]


def _grid_csr(shape, offsets, coef):
    """CSR arrays (int32, int32, float64) of a stencil on a grid, x fastest, columns ascending.
    coef: a number or a tensor of one value per row for each offset."""
    nx, ny, nz = shape
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
    ok = torch.stack([(ix + a >= 0) & (ix + a < nx) & (iy + b >= 0) & (iy + b < ny) &
                      (iz + c >= 0) & (iz + c < nz) for a, b, c in offsets], 1)
    col = torch.stack([i + a + nx * (b + ny * c) for a, b, c in offsets], 1)
    val = torch.stack([torch.as_tensor(v, device="cuda", dtype=F64).expand(n) for v in coef], 1)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = ok.sum(1).cumsum(0)
    return rp.to(torch.int32), col[ok].to(torch.int32), val[ok].contiguous()


def _grid_apply(shape, offsets, coef, u):
    """The stencil applied to u, in torch alone."""
    nx, ny, nz = shape
    v = torch.nn.functional.pad(u.view(nz, ny, nx), (1, 1, 1, 1, 1, 1))
    out = torch.zeros_like(u)
    for (a, b, c), w in zip(offsets, coef):
        out += w * v[1 + c:1 + c + nz, 1 + b:1 + b + ny, 1 + a:1 + a + nx].reshape(-1)
    return out


def _poisson(dim, m, shift=0.0):
    return ((m, m, 1), _OFF2, [-1.0, -1.0, 4.0 + shift, -1.0, -1.0]) if dim == 2 else \
        ((m, m, m), _OFF3, [-1.0, -1.0, -1.0, 6.0 + shift, -1.0, -1.0, -1.0])


def _convdiff(m, peclet, step=None):
    """Upwind convection-diffusion times h^2, cell Peclet number as given, flow along
    (1, 0.5, 0.25); with step, the implicit Euler matrix I + step * that."""
    c = [-1.0, -1.0, -1.0, 6.0, -1.0, -1.0, -1.0]
    for lo, d in ((2, 1.0), (1, 0.5), (0, 0.25)):
        c[lo] -= 2.0 * peclet * d
        c[3] += 2.0 * peclet * d
    if step is not None:
        c = [step * v for v in c]
        c[3] += 1.0
    return (m, m, m), _OFF3, c


def _vardiff(m, g):
    """-div(k grad u) on m^3 cells, k log-normal, harmonic means on the faces."""
    k = torch.exp(0.5 * torch.randn(m ** 3, generator=g, device="cuda", dtype=F64)).view(m, m, m)
    diag = torch.zeros_like(k)
    coef = []
    for a, b, c in _OFF3:
        if (a, b, c) == (0, 0, 0):
            coef.append(None)
            continue
        p = torch.nn.functional.pad(k[None], (1,) * 6, mode="replicate")[0]
        nb = p[1 + c:1 + c + m, 1 + b:1 + b + m, 1 + a:1 + a + m]
        f = 2.0 * k * nb / (k + nb)
        diag += f
        coef.append(-f.reshape(-1))
    coef[3] = diag.reshape(-1)
    return (m, m, m), _OFF3, coef


def _fem(m, g):
    """Triplets of a finite-element-like symmetric matrix on m^3 nodes: edge conductances to the
    26 neighbours (one in eight edges missing) plus a mass term, nodes numbered at random inside
    groups of 64. Row-major order, columns ascending: (rows, columns, values), int64 and float64."""
    n = m ** 3
    i = torch.arange(n, device="cuda")
    ix, iy, iz = i % m, (i // m) % m, i // (m * m)
    perm = torch.argsort(torch.rand(n, generator=g, device="cuda", dtype=F64) + (i // 64).to(F64))
    rows, cols, vals = [], [], []
    diag = _uniform(g, n, 0.05, 0.1)
    for dz in (0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) <= (0, 0, 0):
                    continue
                ok = (ix + dx >= 0) & (ix + dx < m) & (iy + dy >= 0) & (iy + dy < m) & \
                    (iz + dz < m) & (torch.rand(n, generator=g, device="cuda") > 0.125)
                a = i[ok]
                b = a + dx + m * (dy + m * dz)
                w = _uniform(g, a.numel(), 0.2, 1.0)
                diag[a] += w
                diag[b] += w
                rows += [perm[a], perm[b]]
                cols += [perm[b], perm[a]]
                vals += [-w, -w]
    r, c, v = torch.cat(rows + [perm]), torch.cat(cols + [perm]), torch.cat(vals + [diag])
    at = torch.argsort(r * n + c)
    return n, r[at], c[at], v[at]


def _csr_of(n, r, c, v):
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.bincount(r, minlength=n).cumsum(0)
    return rp.to(torch.int32), c.to(torch.int32), v


def _mat(csr, mcol=None):
    rp, ci, va = csr
    n = rp.numel() - 1
    torch.cuda.synchronize()
    h = C.c_void_p()
    check(lib.fasp_gpu_mat_create_device(n, n if mcol is None else mcol, ci.numel(), rp.data_ptr(),
                                         ci.data_ptr(), va.data_ptr(), C.byref(h)), "MAT")
    return sol.MAT(_handle=h)


def _interp(m):
    """CSR arrays of the trilinear interpolation from (m - 1) / 2 to m points a side."""
    mc = (m - 1) // 2
    i = torch.arange(m, device="cuda")
    odd = i % 2 == 1
    c1 = torch.stack([(i - 1) // 2, i // 2], 1)  # odd: one parent; even: two, weight 1/2
    w1 = torch.where(odd[:, None], torch.tensor([1.0, 0.0], device="cuda", dtype=F64), 0.5)
    w1 = torch.where((c1 >= 0) & (c1 < mc), w1, 0.0)
    c1[:, 0] = torch.where(odd, c1[:, 0], i // 2 - 1)
    w1[:, 0] = torch.where(odd, 1.0, torch.where(c1[:, 0] >= 0, 0.5, 0.0))
    c = (c1[:, None, None, :, None, None] * mc + c1[None, :, None, None, :, None]) * mc + \
        c1[None, None, :, None, None, :]
    w = w1[:, None, None, :, None, None] * w1[None, :, None, None, :, None] * \
        w1[None, None, :, None, None, :]
    c, w = c.reshape(m ** 3, 8), w.reshape(m ** 3, 8)
    ok = w > 0
    rp = torch.zeros(m ** 3 + 1, dtype=torch.int64, device="cuda")
    rp[1:] = ok.sum(1).cumsum(0)
    return (rp.to(torch.int32), c[ok].to(torch.int32), w[ok].contiguous()), mc


def _solver(alg, M, precision="fp64", transfers=None, **kw):
    s = sol.configure(alg, relTol=1e-8, absTol=0.0, maxIter=5000, **kw)
    if precision == "mixed":
        s.SetPrecision(capi.MIXED_RELIABLE, innerRelTol=1e-2)
    if transfers:
        s.transfers = {k: (P, None, None) for k, P in enumerate(transfers)}
    s.Setup(M)
    return s


def _problem(case, seed):
    """What the seed decides: the matrix, the vectors."""
    g = _gen(seed)
    f, m = case["family"], case.get("m")
    if f == "step":
        n = m * m
        return {"grid": _poisson(2, m), "p": _uniform(g, n, -1, 1), "r": _uniform(g, n, -1, 1),
                "x": _uniform(g, n)}
    if f == "product":
        if case["kind"] == "fem":
            n, r, c, v = _fem(m, g)
            d = {"csr": _csr_of(n, r, c, v), "rows": r}
        else:
            grid = _vardiff(m, g) if case["kind"] == "var" else _poisson(3, m)
            d = {"csr": _grid_csr(*grid)}
            n = m ** 3
            d["rows"] = torch.repeat_interleave(torch.arange(n, device="cuda"),
                                                d["csr"][0].diff().long())
        return {**d, "x": _uniform(g, n, -1, 1), "b": _uniform(g, n, -1, 1)}
    if f in ("cg", "bicgstab", "gmres", "mgcg"):
        grid = _poisson(case["dim"], m) if f == "cg" else _poisson(3, m) if f == "mgcg" else \
            _convdiff(m, case["peclet"], case.get("step"))
        xs = _uniform(g, grid[0][0] * grid[0][1] * grid[0][2])
        return {"grid": grid, "x": xs, "b": _grid_apply(*grid, xs)}
    if f == "galerkin":
        P, mc = _interp(m)
        return {"csr": _grid_csr(*_vardiff(m, g)), "P": P, "mc": mc}
    if f == "assemble":
        n, r, c, v = _fem(m, g)
        at = torch.randperm(r.numel(), generator=g, device="cuda")
        return {"n": n, "rows": r[at].to(torch.int32), "cols": c[at].to(torch.int32), "vals": v[at],
                "x": _uniform(g, n, -1, 1)}
    if f == "train":
        grid = _vardiff(m, g)
        n = m ** 3
        return {"csr": _grid_csr(*grid), "grid": grid, "b": _uniform(g, n, -1, 1),
                "g": _uniform(g, n, -1, 1)}
    if f == "batch":
        # the grids' sizes belong to the case, the shifts and right-hand sides to the seed
        ms = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1,
                                                           size=case["count"])
        sig = np.random.default_rng(seed).uniform(0.0, 1.0, size=case["count"])
        N = int((ms.astype(np.int64) ** 2).sum())
        return {"ms": ms, "sig": sig,
                "b": torch.randn(case["nrhs"], N, generator=g, device="cuda", dtype=F64)}
    raise ValueError(f)


def prepare(case, seed):
    capi.init(0)
    f = case["family"]
    s = _problem(case, seed)
    s["family"] = f
    if f == "step":
        s["M"] = _mat(_grid_csr(*s["grid"]))
    elif f == "product":
        s["M"] = _mat(s["csr"])
        n = s["M"].nrow
        s["v"] = [_Vec(torch.empty(n, device="cuda", dtype=F64)) for _ in range(3)]
        del s["rows"]
        s["M"].MultTransposeAdd(_Vec(s["x"]), _Vec(s["b"]), s["v"][0])  # keeps the transpose
    elif f in ("cg", "bicgstab", "gmres"):
        s["M"] = _mat(_grid_csr(*s["grid"]))
        kw = dict(maxRestart=30, minRestart=30) if f == "gmres" else {}
        s["S"] = _solver(f, s["M"], case.get("precision", "fp64"), pcd="jacobi", pcdIter=1, **kw)
    elif f == "mgcg":
        s["M"] = _mat(_grid_csr(*s["grid"]))
        m, s["P"] = case["m"], []
        while m > 3 and m % 2 == 1:
            P, mc = _interp(m)
            s["P"].append(_mat(P, mc ** 3))
            m = mc
        sm = dict(maxIter=2, minIter=2, weight=2.0 / 3.0)
        s["S"] = _solver("cg", s["M"], transfers=s["P"], pcd="mg", pcdIter=1, mgLevels=len(s["P"]),
                         mgCycles=1, mgSmooth=sm, mgCoarse=dict(sm, maxIter=40, minIter=40))
    elif f == "galerkin":
        s["A"] = _mat(s["csr"])
        s["PM"] = _mat(s["P"], s["mc"] ** 3)
        nc = s["mc"] ** 3
        # page-locked host arrays for the product, at most 27 entries a row
        s["out"] = [torch.empty(k, dtype=t).pin_memory() for k, t in
                    ((nc + 1, torch.int32), (27 * nc, torch.int32), (27 * nc, F64))]
    elif f == "assemble":
        s["d"] = [_Vec(s[k]) for k in ("rows", "cols", "vals")]
    elif f == "train":
        rp, ci, va = s["csr"]
        s["system"] = SparseSystem(rp.cpu().numpy(), ci.cpu().numpy(), rp.numel() - 1)
        s["va"] = va.requires_grad_(True)
        s["b"].requires_grad_(True)
    elif f == "batch":
        s.update(_batch(s["ms"], s["sig"], case["nrhs"]))
        s["precision"] = capi.FP64 if case["precision"] == "fp64" else capi.MIXED_RELIABLE
    return s


def _batch(ms, sig, nrhs):
    """A batch handle of shifted 2D Poisson systems (block-diagonal CSR on the GPU)."""
    sys_row = np.zeros(len(ms) + 1, np.int64)
    np.cumsum(ms.astype(np.int64) ** 2, out=sys_row[1:])
    start = torch.from_numpy(sys_row).cuda()
    m, sg = torch.from_numpy(ms.astype(np.int64)).cuda(), torch.from_numpy(sig).cuda()
    k = torch.repeat_interleave(torch.arange(len(ms), device="cuda"), m * m)
    i = torch.arange(int(sys_row[-1]), device="cuda")
    mk, loc = m[k], i - start[k]
    ix, iy = loc % mk, loc // mk
    ok = torch.stack([iy > 0, ix > 0, ix >= 0, ix < mk - 1, iy < mk - 1], 1)
    col = torch.stack([i - mk, i - 1, i, i + 1, i + mk], 1)
    one = torch.full_like(sg[k], -1.0)
    val = torch.stack([one, one, 4.0 + sg[k], one, one], 1)
    rp = torch.zeros(i.numel() + 1, dtype=torch.int64, device="cuda")
    rp[1:] = ok.sum(1).cumsum(0)
    arr = [start.to(torch.int32), rp.to(torch.int32), col[ok].to(torch.int32), val[ok].contiguous()]
    torch.cuda.synchronize()
    h = C.c_void_p()
    check(lib.fasp_gpu_batch_create(len(ms), arr[0].data_ptr(), arr[2].numel(), arr[1].data_ptr(),
                                    arr[2].data_ptr(), arr[3].data_ptr(), nrhs, C.byref(h)),
          "batch_create")
    return {"h": _BatchHandle(h), "count": len(ms), "nrhs": nrhs}


class _BatchHandle:
    def __init__(self, h):
        self.h = h

    def __del__(self):
        lib.fasp_gpu_batch_destroy(self.h)


# ---- one pass --------------------------------------------------------------------------

def run(s):
    return _RUN[s["family"]](s)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _run_step(s):
    p, r, x = _Vec(s["p"]), _Vec(s["r"]), _Vec(s["x"])
    q, r1, x1, p1 = (_Vec(torch.empty_like(s["p"])) for _ in range(4))
    s["M"].Apply(p, q)
    rr = r.Dot(r)
    alpha = rr / p.Dot(q)
    x1.WAXPBY(1.0, x, alpha, p)
    r1.WAXPBY(1.0, r, -alpha, q)
    res = r1.Norm2()
    p1.WAXPBY(1.0, r1, res * res / rr, p)
    return x1.t, r1.t, p1.t, res


def _run_product(s):
    y, r, v = s["v"]
    x, b = _Vec(s["x"]), _Vec(s["b"])
    s["M"].Apply(x, y)
    s["M"].Residual(b, x, r)
    s["M"].MultTransposeAdd(x, b, v)
    return y.t, r.t, v.t


def _run_solve(s):
    x, info = torch.zeros_like(s["b"]), capi.Info()
    check(lib.fasp_gpu_solver_solve_async(s["S"].h, s["b"].data_ptr(), x.data_ptr(), C.byref(info),
                                          _stream()), "Solve")
    return x


def _run_galerkin(s):
    R = s["PM"].Transpose()
    Ac = R.Mult(s["A"].Mult(s["PM"]))
    rp, ci, va = s["out"]
    check(lib.fasp_gpu_mat_download(Ac.h, rp.data_ptr(), ci.data_ptr(), va.data_ptr(), None),
          "download")
    return rp, ci[:Ac.nnz], va[:Ac.nnz]


def _run_assemble(s):
    A = sol.MAT.FromCOO(s["n"], s["n"], *s["d"])
    y, d = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    A.Apply(_Vec(s["x"]), _Vec(y))
    check(lib.fasp_gpu_mat_diag(A.h, d.data_ptr()), "GetDiag")
    return y, d


def _run_train(s):
    x = sparse_solve(s["va"], s["b"], s["system"])
    dA, db = torch.autograd.grad(x, (s["va"], s["b"]), s["g"])
    return x.detach(), dA, db


def _run_batch(s):
    x = torch.empty_like(s["b"])
    it = np.zeros(s["count"] * s["nrhs"], np.uint32)
    check(lib.fasp_gpu_batch_solve_async(s["h"].h, s["b"].data_ptr(), x.data_ptr(), 1e-8, 5000,
                                         s["precision"], 0.01, it.ctypes.data, None, _stream()),
          "batch_solve")
    return x


_RUN = {"step": _run_step, "product": _run_product, "cg": _run_solve, "bicgstab": _run_solve,
        "gmres": _run_solve, "mgcg": _run_solve, "galerkin": _run_galerkin,
        "assemble": _run_assemble, "train": _run_train, "batch": _run_batch}


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; an iterative method reads its matrix and
    right-hand side and writes its solution once (what its iterations move is the library's
    affair), and its operations are those of the iterations it needs at the least (about m for
    Jacobi-CG on a grid of m points a side)."""
    f, m = case["family"], case.get("m", 0)
    if f == "step":
        n = m * m
        return {"bytes": 12.0 * 5 * n + 8.0 * 6 * n, "flops": 22.0 * n}
    if f == "product":
        n = float(m ** 3)
        nnz = 23.0 * n if case["kind"] == "fem" else 7.0 * n
        return {"bytes": 12 * nnz + 4 * n + 8 * 5 * n, "flops": 6 * nnz}
    n = float(m ** case.get("dim", 3))
    if f in ("cg", "gmres", "bicgstab", "mgcg"):
        its = {"cg": 2.5 * m, "gmres": 2.5 * m, "bicgstab": 15, "mgcg": 9}[f]
        per = {"cg": 24, "gmres": 90, "bicgstab": 48, "mgcg": 130}[f]
        return {"bytes": 12 * 7 * n + 16 * n, "flops": its * per * n}
    if f == "galerkin":
        return {"bytes": 12 * 7 * n + 12 * 3.375 * n + 12 * 27 * n / 8,
                "flops": 2 * 24 * n + 2 * 40 * n}
    if f == "assemble":
        return {"bytes": 16 * 23 * n + 24 * n, "flops": 46 * n}
    if f == "train":
        return {"bytes": 12 * 7 * n + 8 * 7 * n + 32 * n, "flops": 2 * 5.0 * m * 24 * n}
    mean = (case["lo"] ** 2 + case["lo"] * case["hi"] + case["hi"] ** 2) / 3.0
    N = case["count"] * mean
    return {"bytes": 12 * 5 * N + 16 * N * case["nrhs"], "flops": 60.0 * 20 * N * case["nrhs"]}


# ---- the same in 64 bits, in plain torch -------------------------------------------------

def exact(case, seed):
    s = _problem(case, seed)
    f = case["family"]
    if f == "step":
        p, r, x = s["p"], s["r"], s["x"]
        q = _grid_apply(*s["grid"], p)
        rr = r @ r
        a = rr / (p @ q)
        x1, r1 = x + a * p, r - a * q
        res = torch.linalg.vector_norm(r1)
        return x1, r1, r1 + (res * res / rr) * p, float(res)
    if f == "product":
        rows, ci, va = s["rows"], s["csr"][1].long(), s["csr"][2]
        x, b = s["x"], s["b"]
        y = torch.zeros_like(x).index_add_(0, rows, va * x[ci])
        return y, b - y, b.index_add(0, ci, va * x[rows])
    if f in ("cg", "bicgstab", "gmres", "mgcg"):
        return s["x"]  # b was made from it
    if f == "galerkin":
        n, nc = case["m"] ** 3, s["mc"] ** 3
        P = s["P"]
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), P[0].diff().long())
        at = torch.argsort(P[1].long() * n + rows)
        R = (*_csr_of(nc, P[1].long()[at], rows[at], P[2][at]),)
        return None, None, _mult(R, _mult(s["csr"], P, nc), nc)[2]
    if f == "assemble":
        r, c = s["rows"].long(), s["cols"].long()
        y = torch.zeros_like(s["x"]).index_add_(0, r, s["vals"] * s["x"][c])
        d = torch.zeros_like(y)
        on = r == c
        d[r[on]] = s["vals"][on]
        return y, d
    if f == "train":
        x, lam = _cg(s["grid"], s["b"]), _cg(s["grid"], s["g"])  # the matrix is symmetric
        rows = torch.repeat_interleave(torch.arange(x.numel(), device="cuda"),
                                       s["csr"][0].diff().long())
        return x, -lam[rows] * x[s["csr"][1].long()], lam
    x, at = torch.empty_like(s["b"]), 0
    for m, sg in zip(s["ms"].tolist(), s["sig"].tolist()):  # sine transforms solve each system
        k = torch.arange(1, m + 1, device="cuda", dtype=F64)
        T = torch.sin(math.pi / (m + 1) * k[:, None] * k) * math.sqrt(2.0 / (m + 1))
        lam = 2.0 - 2.0 * torch.cos(math.pi / (m + 1) * k)
        b = s["b"][:, at:at + m * m].view(-1, m, m)
        x[:, at:at + m * m] = (T @ ((T @ b @ T) / (lam[:, None] + lam + sg)) @ T).view(-1, m * m)
        at += m * m
    return x


def _mult(A, B, ncol):
    """CSR arrays of A B: the columns of a row in the order in which the row meets them."""
    rp, ci, va = A
    rows = torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp.diff().long())
    cnt = B[0].diff().long()[ci.long()]
    e = torch.repeat_interleave(torch.arange(ci.numel(), device="cuda"), cnt)
    k = torch.arange(e.numel(), device="cuda") - (cnt.cumsum(0) - cnt)[e] + B[0].long()[ci.long()[e]]
    key, grp = torch.unique(rows[e] * ncol + B[1].long()[k], return_inverse=True)
    val = torch.zeros(key.numel(), device="cuda", dtype=F64).index_add_(0, grp, va[e] * B[2][k])
    first = torch.full_like(key, e.numel())
    first.scatter_reduce_(0, grp, torch.arange(e.numel(), device="cuda"), "amin")
    at = torch.argsort(first)  # rows come in order, and so do their first meetings
    return _csr_of(rp.numel() - 1, (key // ncol)[at], (key % ncol)[at], val[at])


def _cg(grid, b):
    """Jacobi-CG in torch, to the rounding of 64 bits."""
    d = 1.0 / grid[2][3]
    x, r = torch.zeros_like(b), b.clone()
    z = d * r
    p, rz, stop = z.clone(), r @ z, 1e-28 * (b @ b)
    for it in range(3000):
        q = _grid_apply(*grid, p)
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        z = d * r
        rz, old = r @ z, rz
        p = z + (rz / old) * p
        if it % 20 == 19 and bool(r @ r < stop):
            break
    return x
