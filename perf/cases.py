"""The work this library is measured by: its solves, its smoothing and triangular-solve kernels, its assembly.

Every case goes through the public entry points of ``fem_gb300.lina`` (the C ABI of include/lina_gpu.h) on the
systems of ``fem_gb300.problems``: P1 Poisson and degraded plane-strain elasticity on m x m grids, the phase-field
damage matrix, unstructured batches, the adjoint pair.  Matrices, hierarchies and factorisations are what a
program sets up once and keeps, so a handle is shared by the states of one size; right-hand sides, start vectors,
moduli and matrix values come from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fem_gb300 import lina, problems


def listed():
    return [
        # the smallest call: one product of a 33 x 33 grid, where the launch and the wait are the time
        {"name": "spmv_poisson33_f64", "kind": "spmv", "matrix": "poisson", "m": 33, "precision": "f64"},
        # one FP32 smoother sweep of the 2.1M-dof matrix, the bandwidth-bound half of every mixed solve
        {"name": "jacobi_elast1025_f32", "kind": "jacobi", "matrix": "elasticity", "m": 1025, "precision": "f32"},
        # one preconditioner application on a small hierarchy of an odd size (a caller's own Krylov loop)
        {"name": "vcycle_elast97_f64", "kind": "vcycle", "matrix": "elasticity", "m": 97, "smoother": "jacobi"},
        # the scalar workload: FP64, aggressive coarsening, multicolour SOR, the reference's stopping rule
        {"name": "pcg_poisson257_f64", "kind": "pcg", "matrix": "poisson", "m": 257, "precision": "f64"},
        # the headline workload: mixed-precision solve of 2.1M dofs
        {"name": "pcg_elast1025_mixed", "kind": "pcg", "matrix": "elasticity", "m": 1025, "precision": "mixed"},
        # the plain FP64 solve at an ordinary, odd size
        {"name": "pcg_elast225_f64", "kind": "pcg", "matrix": "elasticity", "m": 225, "precision": "f64"},
        # ILU(0) application on the damage workload's matrix, in the precision its minimiser uses
        {"name": "ilu_damage1025_f32", "kind": "ilu", "m": 1025, "precision": "f32"},
        # the same in FP64 at a ragged size
        {"name": "ilu_damage389_f64", "kind": "ilu", "m": 389, "precision": "f64"},
        # the linear solve of one Newton step of the damage minimiser: new values, refactorisation, BiCGStab
        {"name": "newton_damage513", "kind": "newton", "m": 513, "precision": "f32"},
        # uneven unstructured systems solved together
        {"name": "segbatch_16", "kind": "segbatch", "count": 16, "lo": 4000, "hi": 120000, "plan": 0},
        # material identification: forward and adjoint solve and the per-element gradient, host arrays
        {"name": "adjoint_257", "kind": "adjoint", "m": 257},
        # reassembly of the 2.1M-dof matrix for new moduli
        {"name": "assemble_elast1025", "kind": "assemble", "matrix": "elasticity", "m": 1025},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["spmv", "jacobi", "vcycle", "pcg", "ilu", "newton", "segbatch", "adjoint", "assemble"])
    matrix = rng.choice(["poisson", "elasticity"])
    if kind in ("spmv", "jacobi"):
        return {"kind": kind, "matrix": matrix, "m": size(17, 1025), "precision": rng.choice(["f64", "f32"])}
    if kind == "vcycle":
        return {"kind": kind, "matrix": matrix, "m": size(33, 385), "smoother": rng.choice(["jacobi", "sor"])}
    if kind == "pcg":
        if matrix == "poisson":
            return {"kind": kind, "matrix": matrix, "m": size(33, 513), "precision": "f64"}
        return {"kind": kind, "matrix": matrix, "m": size(33, 513), "precision": rng.choice(["f64", "mixed"])}
    if kind == "ilu":
        return {"kind": kind, "m": size(65, 1025), "precision": rng.choice(["f64", "f32"])}
    if kind == "newton":
        return {"kind": kind, "m": size(65, 513), "precision": rng.choice(["f64", "f32"])}
    if kind == "segbatch":
        return {"kind": kind, "count": rng.randint(4, 16), "lo": 4000, "hi": size(20000, 120000),
                "plan": rng.randint(1, 99)}
    if kind == "adjoint":
        return {"kind": kind, "m": size(33, 257)}
    return {"kind": kind, "matrix": matrix, "m": size(65, 1025)}


# ------------------------------------------------------------------------------------------------ inputs
class _Vector:
    """A torch tensor where the binding takes a device array."""

    def __init__(self, t):
        self.t = t
        self.ptr = t.data_ptr()
        self.n = t.numel()


class _Memory:
    """The library's device memory as a torch tensor."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 2}


def _uniform(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (2 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1).to(dtype)


@functools.lru_cache(maxsize=2)
def _system(matrix, m):
    if matrix == "poisson":
        return problems.poisson_p1(m)
    if matrix == "damage":
        return problems.at2_damage(m)
    return problems.elasticity_p1(m)


@functools.lru_cache(maxsize=2)
def _batch(count, lo, hi, plan):
    return [problems.batch_system(*p) for p in problems.batch_plan(count, plan, lo, hi)]


def _rows(s):
    """Row index of every stored entry."""
    return np.repeat(np.arange(s.n), np.diff(s.indptr))


def _load(s, seed):
    """A right-hand side for s: its own plus a seeded one, zero on the rows whose value is prescribed."""
    free = torch.from_numpy(np.diff(s.indptr) > 1).cuda()
    own = torch.from_numpy(s.b).cuda()
    scale = float(np.abs(s.b).max()) or 1.0
    return own + torch.where(free, scale * _uniform(s.n, seed), torch.zeros_like(own))


# ------------------------------------------------------------------------------------------------ handles
@functools.lru_cache(maxsize=1)
def _matrix(matrix, m):
    s = _system(matrix, m)
    return lina.Matrix(s.n, s.indptr, s.indices, s.data)


@functools.lru_cache(maxsize=1)
def _hierarchy(matrix, m, precision, smoother):
    s = _system(matrix, m)
    prec = lina.PREC_MIXED if precision == "mixed" else lina.PREC_FP64
    if smoother == "sor":
        smooth, omega = lina.SMOOTHER_MC_SOR, 1.0
    else:
        smooth, omega = lina.SMOOTHER_JACOBI, 0.6
    if matrix == "poisson":
        return lina.AMG.from_system(s, depth=min(6, problems.batch_depth(s.n)), coarsening=lina.AGGRESSIVE,
                                    smoother=smooth, omega=omega, precision=prec)
    return lina.AMG.from_system(s, depth=problems.batch_depth(s.n), coarsening=lina.STANDARD, matrix_tol=0.1,
                                smoother=smooth, omega=omega, precision=prec)


@functools.lru_cache(maxsize=1)
def _ilu(m):
    s = _system("damage", m)
    return lina.ILU(s.n, s.indptr, s.indices, s.data)


@functools.lru_cache(maxsize=1)
def _newton(m):
    s = _system("damage", m)
    return lina.Matrix(s.n, s.indptr, s.indices, s.data), lina.ILU(s.n, s.indptr, s.indices, s.data)


@functools.lru_cache(maxsize=1)
def _segbatch(count, lo, hi, plan):
    amgs = [lina.AMG.from_system(s, depth=problems.batch_depth(s.n), coarsening=lina.STANDARD,
                                 smoother=lina.SMOOTHER_MC_SOR, omega=1.0, precision=lina.PREC_MIXED, matrix_tol=0.3)
            for s in _batch(count, lo, hi, plan)]
    return lina.SegmentedBatch(amgs)


def _adjoint_inputs(m, seed):
    case = problems.adjoint_case(m, seed=0, n_sensors=min(256, m * (m - 2) // 4))
    xy, tri, fd, fv = problems.elastic_mesh(m)
    rng = np.random.default_rng(seed)
    # observed displacements of a stretched plate with measurement noise, moduli near the handle's
    nodes = case["sensor_dof"][:len(case["sensor_dof"]) // 2]
    target = np.concatenate([np.zeros(len(nodes)), 1e-3 * xy[nodes, 1]])
    young = case["young"] * np.exp(0.1 * rng.standard_normal(len(case["young"])))
    return case, xy, tri, fd, fv, target, young


@functools.lru_cache(maxsize=1)
def _adjoint(m):
    case, xy, tri, fd, fv, target, _ = _adjoint_inputs(m, 0)
    return lina.ElasticAdjoint(xy, tri, 0.3, fd, fv, case["sensor_dof"], target, case["young"],
                               depth=max(2, problems.batch_depth(2 * m * m) - 1), precision=lina.PREC_MIXED,
                               coarsening=lina.STANDARD)


def _mesh(matrix, m):
    xy, tri, fd, fv = problems.elastic_mesh(m)
    if matrix == "elasticity":
        return lina.P1_ELASTIC, xy, tri, fd, fv
    edge = np.nonzero((xy[:, 0] == 0) | (xy[:, 0] == 1) | (xy[:, 1] == 0) | (xy[:, 1] == 1))[0].astype(np.int32)
    return lina.P1_LAPLACE, xy, tri, edge, np.zeros(len(edge))


@functools.lru_cache(maxsize=1)
def _assembly(matrix, m):
    kind, xy, tri, fd, fv = _mesh(matrix, m)
    return lina.P1Assembly(kind, xy, tri, nu=0.3, fixed_dof=fd, fixed_val=fv)


def _moduli(m, seed):
    """Lognormal per-element coefficients."""
    return torch.exp(0.5 * torch.randn(2 * (m - 1) ** 2, dtype=torch.float64, device="cuda",
                                       generator=torch.Generator(device="cuda").manual_seed(seed)))


def _newton_values(s, seed):
    """The scaled Newton matrix of an iterate in a box: D A D + diag(v) with D in (0.2, 1) and v >= 0."""
    rng = np.random.default_rng(seed)
    d = np.sqrt(rng.uniform(0.04, 1.0, s.n))
    rows = _rows(s)
    val = s.data * d[rows] * d[s.indices]
    diag = rows == s.indices
    val[diag] += rng.uniform(0.0, 0.5, s.n) * np.abs(s.data[diag])
    return val


# ------------------------------------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind, s = case["kind"], None
    st = {"kind": kind}
    if kind in ("spmv", "jacobi"):
        s = _system(case["matrix"], case["m"])
        dt = torch.float32 if case["precision"] == "f32" else torch.float64
        st["precision"] = lina.PREC_MIXED if case["precision"] == "f32" else lina.PREC_FP64
        st["A"] = _matrix(case["matrix"], case["m"])
        st["x"] = _Vector(_uniform(s.n, seed, dt))
        st["b"] = _Vector(_uniform(s.n, seed + 1000003, dt))
        st["y"] = _Vector(torch.empty(s.n, dtype=dt, device="cuda"))
    elif kind == "vcycle":
        s = _system(case["matrix"], case["m"])
        st["amg"] = _hierarchy(case["matrix"], case["m"], "f64", case["smoother"])
        st["r"] = _Vector(_load(s, seed))
        st["z"] = _Vector(torch.empty(s.n, dtype=torch.float64, device="cuda"))
    elif kind == "pcg":
        s = _system(case["matrix"], case["m"])
        poisson = case["matrix"] == "poisson"
        st["amg"] = _hierarchy(case["matrix"], case["m"], case["precision"], "sor" if poisson else "jacobi")
        st["b"] = _Vector(_load(s, seed))
        st["x"] = _Vector(torch.empty(s.n, dtype=torch.float64, device="cuda"))
        st["how"] = (dict(tol=1e-8, stop=lina.STOP_REFERENCE, flags=lina.PCG_NORMALIZE | lina.PCG_FINAL_PRECON)
                     if poisson else dict(tol=1e-10, stop=lina.STOP_RELATIVE))
    elif kind == "ilu":
        s = _system("damage", case["m"])
        st["precision"] = lina.PREC_MIXED if case["precision"] == "f32" else lina.PREC_FP64
        st["ilu"] = _ilu(case["m"])
        st["r"] = _Vector(_uniform(s.n, seed))
        st["z"] = _Vector(torch.empty(s.n, dtype=torch.float64, device="cuda"))
    elif kind == "newton":
        s = _system("damage", case["m"])
        st["precision"] = lina.PREC_MIXED if case["precision"] == "f32" else lina.PREC_FP64
        st["A"], st["ilu"] = _newton(case["m"])
        st["val"] = _Vector(torch.from_numpy(_newton_values(s, seed)).cuda())
        st["b"] = _Vector(_uniform(s.n, seed))
        st["x"] = _Vector(torch.empty(s.n, dtype=torch.float64, device="cuda"))
    elif kind == "segbatch":
        spec = (case["count"], case["lo"], case["hi"], case["plan"])
        st["batch"] = _segbatch(*spec)
        st["b"] = [_Vector(_load(s, seed + 101 * i)) for i, s in enumerate(_batch(*spec))]
        st["x"] = [torch.empty(b.n, dtype=torch.float64, device="cuda") for b in st["b"]]
    elif kind == "adjoint":
        st["adj"] = _adjoint(case["m"])
        st["young"] = _adjoint_inputs(case["m"], seed)[-1]
    else:
        st["p1"] = _assembly(case["matrix"], case["m"])
        st["coef"] = _moduli(case["m"], seed)
    torch.cuda.synchronize()  # the library works on streams of its own
    return st


def _ok(rc):
    if rc != 0:
        raise RuntimeError(f"the call failed ({rc}): {lina.last_error()}")


def run(st):
    kind, L = st["kind"], lina.lib()
    if kind == "spmv":
        st["A"].spmv_device(st["x"], st["y"], st["precision"])
        return st["y"].t
    if kind == "jacobi":  # one sweep: the result is in the second buffer, x stays as it is
        st["A"].jacobi_device(st["b"], st["x"], st["y"], 0.6, 1, st["precision"])
        return st["y"].t
    if kind == "vcycle":
        _ok(L.lina_gpu_vcycle(st["amg"].h, st["r"].ptr, st["z"].ptr))
        return st["z"].t
    if kind == "pcg":
        st["amg"].pcg_device(st["b"], st["x"], max_iter=1000, **st["how"])
        return st["x"].t
    if kind == "ilu":
        _ok(L.lina_gpu_ilu_apply(st["ilu"].h, st["precision"], st["r"].ptr, st["z"].ptr))
        return st["z"].t
    if kind == "newton":
        val = lina.C.cast(st["val"].ptr, lina.C.POINTER(lina.C.c_double))
        _ok(L.lina_gpu_matrix_update_values(st["A"].h, val, lina.PCG_DEVICE_PTRS))
        _ok(L.lina_gpu_ilu_refactor(st["ilu"].h, val, lina.PCG_DEVICE_PTRS))
        info = lina.SolveInfo()
        _ok(L.lina_gpu_bicgstab(st["A"].h, st["ilu"].h, st["precision"], st["b"].ptr, st["x"].ptr, 1e-10, 1000,
                                lina.PCG_DEVICE_PTRS, info))
        return st["x"].t
    if kind == "segbatch":
        k = len(st["b"])
        bp = (lina.C.c_void_p * k)(*[b.ptr for b in st["b"]])
        xp = (lina.C.c_void_p * k)(*[x.data_ptr() for x in st["x"]])
        infos = (lina.SolveInfo * k)()
        _ok(L.lina_gpu_segbatch_solve(st["batch"].h, bp, xp, 1e-10, 1000, lina.PCG_DEVICE_PTRS, infos))
        return list(st["x"])
    if kind == "adjoint":
        u, loss, _ = st["adj"].forward(st["young"])
        grad, lam, _ = st["adj"].backward()
        return {"u": u, "loss": loss, "grad": grad, "lam": lam}
    _ok(L.lina_gpu_p1_assemble(st["p1"].h, st["coef"].data_ptr(), lina.PCG_DEVICE_PTRS))
    val, b = st["p1"].device_values()
    return {"values": torch.as_tensor(_Memory(val, st["p1"].nnz), device="cuda"),
            "b": torch.as_tensor(_Memory(b, st["p1"].n), device="cuda")}


def work(case):
    """Bytes and FP operations of one pass: operands read once, results written once per operation of the method.

    A solve is counted as its method's operations: per iteration of AMG-PCG four passes over every level's matrix
    and the Krylov product and vectors (per unknown of these hierarchies 2.4 kB in mixed precision and 4.3 kB in
    FP64 for elasticity, 0.9 kB for the scalar problem), for the usual number of iterations.
    """
    kind = case["kind"]
    if kind == "segbatch":
        n = sum(p[1] for p in problems.batch_plan(case["count"], case["plan"], case["lo"], case["hi"]))
        return {"bytes": 40 * 1000.0 * n, "flops": 40 * 300.0 * n}
    m = case["m"]
    nodes = m * m
    elastic = case.get("matrix") == "elasticity" or kind == "adjoint"
    n = nodes * (2 if elastic else 1)
    nnz = n * (14 if elastic else 7)
    w = 4 if case.get("precision") == "f32" else 8
    if kind == "spmv":
        return {"bytes": (w + 4.0) * nnz + 2.0 * w * n, "flops": 2.0 * nnz}
    if kind == "jacobi":
        return {"bytes": (w + 4.0) * nnz + 4.0 * w * n, "flops": 2.0 * nnz + 4.0 * n}
    if kind == "vcycle":
        return {"bytes": (4.0 if elastic else 0.75) * 1e3 * n, "flops": (700.0 if elastic else 120.0) * n}
    if kind == "pcg":
        per, its = (900.0, 13) if not elastic else (2400.0, 38) if case["precision"] == "mixed" else (4300.0, 40)
        return {"bytes": per * its * n, "flops": per * its * n / 6}
    if kind == "ilu":  # off-diagonal entries once; per triangular solve 1/diagonal, right-hand side and result
        return {"bytes": (w + 4.0) * (nnz - n) + 5.0 * w * n, "flops": 2.0 * nnz}
    if kind == "newton":  # the refactorisation, then about 20 applications and products
        return {"bytes": 24.0 * nnz + 20 * ((w + 4.0) * nnz + 12.0 * nnz + 100.0 * n), "flops": 80.0 * nnz}
    if kind == "adjoint":
        return {"bytes": 2 * 60 * 2400.0 * n, "flops": 2 * 60 * 400.0 * n}
    ne = 2 * (m - 1) ** 2  # coefficient, vertices and geometry of every element, the values and b
    return {"bytes": (8.0 + 12.0 + 56.0) * ne + 8.0 * (nnz + n), "flops": (72.0 if elastic else 18.0) * ne}


# ------------------------------------------------------------------------------------------------ 64-bit values
def _csr(s, val=None):
    return torch.sparse_csr_tensor(torch.from_numpy(s.indptr.astype(np.int64)), torch.from_numpy(s.indices.astype(np.int64)),
                                   torch.from_numpy(s.data if val is None else val), size=(s.n, s.n)).cuda()


def _solve(A, diag, b, limit=60000):
    """A x = b, symmetric positive definite: Jacobi-preconditioned CG, restarted from the true residual until
    that no longer falls."""
    x = torch.zeros_like(b)
    best = math.inf
    dinv = 1.0 / diag
    done = 0
    for _ in range(8):
        r = b - A @ x
        norm = float(r.norm())
        if norm == 0.0 or norm > 0.2 * best or done >= limit:
            break
        best = norm
        z = dinv * r
        p, rz, d = z.clone(), r @ z, torch.zeros_like(b)
        while done < limit:
            for _ in range(50):
                q = A @ p
                a = rz / (p @ q)
                d = d + a * p
                r = r - a * q
                z = dinv * r
                rz, old = r @ z, rz
                p = z + (rz / old) * p
            done += 50
            if float(r.norm()) < 1e-13 * norm:
                break
        x = x + d
    return x


def _spd(s, b, val=None):
    data = s.data if val is None else val
    rows = _rows(s)
    at = rows == s.indices
    return _solve(_csr(s, val), torch.from_numpy(data[at]).cuda(), b)


def _diagonals(s, m):
    """The seven diagonals of a structured damage matrix, d[(dr, dc)][r, c]."""
    rows = _rows(s)
    dr = s.indices // m - rows // m
    dc = s.indices % m - rows % m
    d = {}
    for o in ((-1, -1), (-1, 0), (0, -1), (0, 0), (0, 1), (1, 0), (1, 1)):
        d[o] = np.zeros((m, m))
        at = (dr == o[0]) & (dc == o[1])
        d[o].ravel()[rows[at]] = s.data[at]
    return d


def _ilu_apply(s, m, r):
    """U^-1 L^-1 r with ILU(0) factors (U with unit diagonal), anti-diagonal by anti-diagonal."""
    f = _diagonals(s, m)
    low, up = [(-1, -1), (-1, 0), (0, -1)], [(0, 1), (1, 0), (1, 1)]
    inside = lambda i, j: (i >= 0) & (i < m) & (j >= 0) & (j < m)  # noqa: E731

    def at(a, i, j):
        return np.where(inside(i, j), a[np.clip(i, 0, m - 1), np.clip(j, 0, m - 1)], 0.0)

    y = np.zeros((m, m))
    rhs = r.reshape(m, m)
    fronts = []
    for k in range(2 * m - 1):
        i = np.arange(max(0, k - m + 1), min(k, m - 1) + 1)
        fronts.append((i, k - i))
    for i, j in fronts:
        v = {o: f[o][i, j].copy() for o in f}
        for a in low:  # in ascending column order: the entry is final when its turn comes
            for b in up:
                o = (a[0] + b[0], a[1] + b[1])
                if o in v:
                    v[o] -= v[a] * at(f[b], i + a[0], j + a[1])
        for b in up:
            v[b] = v[b] / v[(0, 0)]
        for o in f:
            f[o][i, j] = v[o]
        y[i, j] = (rhs[i, j] - sum(v[a] * at(y, i + a[0], j + a[1]) for a in low)) / v[(0, 0)]
    z = np.zeros((m, m))
    for i, j in reversed(fronts):
        z[i, j] = y[i, j] - sum(f[b][i, j] * at(z, i + b[0], j + b[1]) for b in up)
    return torch.from_numpy(z.ravel())


def _elements(m, elastic, xy, tri):
    """Unit-coefficient P1 element matrices and the global unknowns of each element."""
    x, y = xy[tri, 0], xy[tri, 1]
    b = np.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], axis=1)
    c = np.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], axis=1)
    area = 0.5 * np.abs((x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0]))
    if not elastic:
        return (b[:, :, None] * b[:, None, :] + c[:, :, None] * c[:, None, :]) / (4 * area)[:, None, None], tri
    nu = 0.3
    B = np.zeros((len(tri), 3, 6))
    B[:, 0, 0:3], B[:, 1, 3:6], B[:, 2, 0:3], B[:, 2, 3:6] = b, c, c, b
    B /= (2 * area)[:, None, None]
    D = np.array([[1 - nu, nu, 0], [nu, 1 - nu, 0], [0, 0, (1 - 2 * nu) / 2]]) / ((1 + nu) * (1 - 2 * nu))
    return np.matmul(B.transpose(0, 2, 1), D @ B) * area[:, None, None], np.concatenate([tri, tri + len(xy)], axis=1)


def _assembled(m, elastic, xy, tri, fd, fv, coef):
    """Row pointers, columns, values and right-hand side with the prescribed unknowns eliminated."""
    ke, dofs = _elements(m, elastic, xy, tri)
    n = len(xy) * (2 if elastic else 1)
    v = torch.from_numpy(ke).cuda() * coef[:, None, None]
    g = torch.from_numpy(dofs.astype(np.int64)).cuda()
    k = g.shape[1]
    at = torch.stack([g[:, :, None].expand(-1, k, k).reshape(-1), g[:, None, :].expand(-1, k, k).reshape(-1)])
    A = torch.sparse_coo_tensor(at, v.reshape(-1), (n, n)).coalesce()
    (row, col), val = A.indices(), A.values()
    fixed = torch.zeros(n, dtype=torch.bool, device="cuda")
    known = torch.zeros(n, dtype=torch.float64, device="cuda")
    where = torch.from_numpy(fd.astype(np.int64)).cuda()
    fixed[where] = True
    known[where] = torch.from_numpy(np.asarray(fv, dtype=np.float64)).cuda()
    b = torch.where(fixed, known, -torch.zeros_like(known).index_add_(0, row, val * known[col]))
    own = fixed[row] & (row == col)
    keep = (~fixed[row] & ~fixed[col]) | own
    val = torch.where(own, torch.ones_like(val), val)
    row, col, val = row[keep], col[keep], val[keep]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return ptr, col, val, b, row == col


def exact(case, seed):
    kind = case["kind"]
    if kind in ("spmv", "jacobi"):
        s = _system(case["matrix"], case["m"])
        dt = torch.float32 if case["precision"] == "f32" else torch.float64
        x = _uniform(s.n, seed, dt).double()
        Ax = _csr(s) @ x
        if kind == "spmv":
            return Ax
        b = _uniform(s.n, seed + 1000003, dt).double()
        diag = torch.from_numpy(s.data[_rows(s) == s.indices]).cuda()
        return x + 0.6 / diag * (b - Ax)
    if kind == "pcg":
        s = _system(case["matrix"], case["m"])
        return _spd(s, _load(s, seed)) if s.n <= 160000 else None
    if kind == "ilu":
        s = _system("damage", case["m"])
        return _ilu_apply(s, case["m"], _uniform(s.n, seed).cpu().numpy())
    if kind == "newton":
        s = _system("damage", case["m"])
        return _spd(s, _uniform(s.n, seed), _newton_values(s, seed))
    if kind == "segbatch":
        systems = _batch(case["count"], case["lo"], case["hi"], case["plan"])
        return [_spd(s, _load(s, seed + 101 * i)) if s.n <= 30000 else None for i, s in enumerate(systems)]
    if kind == "adjoint":
        m = case["m"]
        c, xy, tri, fd, fv, target, young = _adjoint_inputs(m, seed)
        E = torch.from_numpy(young).cuda()
        ptr, col, val, b, own = _assembled(m, True, xy, tri, fd, fv, E)
        A = torch.sparse_csr_tensor(ptr, col, val, size=(len(b), len(b)))
        u = _solve(A, val[own], b)
        at = torch.from_numpy(c["sensor_dof"].astype(np.int64)).cuda()
        miss = u[at] - torch.from_numpy(target).cuda()
        lam = _solve(A, val[own], torch.zeros_like(u).index_put_((at,), miss))
        ke, dofs = _elements(m, True, xy, tri)
        g = torch.from_numpy(dofs.astype(np.int64)).cuda()
        grad = -torch.einsum("ea,eab,eb->e", lam[g], torch.from_numpy(ke).cuda(), u[g])
        return {"u": u, "loss": 0.5 * float(miss @ miss), "grad": grad, "lam": lam}
    if kind == "assemble":
        _, xy, tri, fd, fv = _mesh(case["matrix"], case["m"])
        _, _, val, b, _ = _assembled(case["m"], case["matrix"] == "elasticity", xy, tri, fd, fv,
                                     _moduli(case["m"], seed))
        return {"values": val, "b": b}
    return None
