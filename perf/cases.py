"""Performance cases of the assembly + preconditioned-CG path.

Each case is one call (or one short sequence of calls) that a user's program
makes again and again on a mesh whose topology it keeps:

* ``solve``: assemble and solve a constrained system for new geometry,
  coefficients and sources (``Problem.solve_device`` with arrays in HBM, or
  ``Problem.solve`` with host arrays), P1 triangles, tetrahedral Lagrange of
  degree 1 to 4 and Nedelec of order 1 and 2, mixed precision or FP64;
* ``assemble``: assemble the constrained operator and right-hand side and apply
  the operator once, as a caller with its own outer iteration does
  (``ffg_problem_assemble``, ``ffg_problem_system_arrays``,
  ``ffg_problem_sell_spmv``), FP64 or 3xTF32 tensor-core contraction;
* ``batch``: many independent systems of different sizes in one
  ``solve_batch`` call, as the serving loop issues them;
* ``csc`` / ``jvp`` / ``vjp``: the drop-in host-array assembly of a Lagrange
  stiffness + mass matrix and its forward and reverse mode, which take a new
  mesh on every call.

Meshes are Kuhn boxes and unit-square triangulations with interior vertices
jittered by 0.1 h, coefficients lognormal per cell (Nedelec: uniform in
[0.5, 2]), sources a few random low-degree trigonometric modes.
``exact`` restates the discretisations in FP64 torch: element matrices by
quadrature, numbering by first appearance, and CG far past the solver's
tolerance.
"""
import ctypes
import itertools
import math

import numpy as np
import torch

import fortfem_b200 as ff
from fortfem_b200 import _capi as K
from fortfem_b200.api import solve_batch

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest everyday 2-D problem (64 x 64 squares): latency counts
        {"name": "p1_square_64", "kind": "solve", "family": "p1", "nx": 64, "ny": 64,
         "precision": "mixed", "host": False},
        # an ordinary 2-D problem of odd size
        {"name": "p1_square_301x287", "kind": "solve", "family": "p1", "nx": 301, "ny": 287,
         "precision": "mixed", "host": False},
        # a small 3-D problem in the reference's precision, host arrays in and out
        {"name": "p2_box_10_fp64_host", "kind": "solve", "family": "lagrange", "degree": 2,
         "nx": 10, "ny": 9, "nz": 11, "precision": "fp64", "host": True},
        # an ordinary 3-D problem of odd size
        {"name": "p2_box_21", "kind": "solve", "family": "lagrange", "degree": 2, "nx": 21,
         "ny": 20, "nz": 23, "precision": "mixed", "host": False},
        # the largest 3-D problem: the repository's benchmark size
        {"name": "p2_box_48", "kind": "solve", "family": "lagrange", "degree": 2, "nx": 48,
         "ny": 48, "nz": 48, "precision": "mixed", "host": False},
        # higher order in FP64, loads with the solver entry's default quadrature
        {"name": "p3_box_14_fp64", "kind": "solve", "family": "lagrange", "degree": 3, "nx": 14,
         "ny": 15, "nz": 14, "precision": "fp64", "host": False},
        # a curl-curl + mass solve at the lowest order
        {"name": "nedelec1_box_15", "kind": "solve", "family": "nedelec", "degree": 1, "nx": 15,
         "ny": 15, "nz": 16, "precision": "mixed", "host": False},
        # high-order edge elements assembled for a caller's own iteration (24^3 is the
        # benchmark's mesh), in FP64
        {"name": "nedelec3_assemble_24", "kind": "assemble", "family": "nedelec", "degree": 3,
         "nx": 24, "ny": 24, "nz": 24, "assembly": "fp64"},
        # the same with the tensor-core contraction
        {"name": "nedelec4_assemble_17_tf32", "kind": "assemble", "family": "nedelec",
         "degree": 4, "nx": 17, "ny": 16, "nz": 17, "assembly": "tf32x3"},
        # the highest order, on the stress case's mesh size
        {"name": "nedelec6_assemble_12", "kind": "assemble", "family": "nedelec", "degree": 6,
         "nx": 12, "ny": 12, "nz": 12, "assembly": "fp64"},
        # one batch of the serving loop: small systems of both families
        {"name": "batch_mixed_12", "kind": "batch", "count": 12, "p1_min": 32, "p1_max": 170,
         "p2_min": 8, "p2_max": 14, "mode": "cta_per_system"},
        # reverse mode through the drop-in entry (shape derivatives of an energy)
        {"name": "p2_vjp_16", "kind": "vjp", "family": "lagrange", "degree": 2, "nx": 16,
         "ny": 16, "nz": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, n):
    return {"nx": n, "ny": max(2, n + rng.randint(-2, 2)), "nz": max(2, n + rng.randint(-2, 2))}


def draw(rng):
    kind = rng.choice(["p1", "p1", "lagrange", "lagrange", "lagrange", "nedelec", "assemble",
                       "assemble", "batch", "host"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "p1":
        n = _log_int(rng, 24, 420)
        return {"kind": "solve", "family": "p1", "nx": n, "ny": max(8, n + rng.randint(-15, 15)),
                "precision": precision, "host": rng.random() < 0.25}
    if kind == "lagrange":
        p = rng.choice([1, 2, 2, 3, 4])
        n = _log_int(rng, 6, {1: 60, 2: 38, 3: 20, 4: 13}[p])
        return dict({"kind": "solve", "family": "lagrange", "degree": p}, **_ragged(rng, n),
                    precision=precision, host=rng.random() < 0.25)
    if kind == "nedelec":
        p = rng.choice([1, 1, 2])
        n = _log_int(rng, 5, {1: 18, 2: 7}[p])
        return dict({"kind": "solve", "family": "nedelec", "degree": p}, **_ragged(rng, n),
                    precision=precision, host=False)
    if kind == "assemble":
        p = rng.choice([1, 2, 3, 4, 5, 6])
        n = _log_int(rng, 4, {1: 32, 2: 28, 3: 24, 4: 17, 5: 13, 6: 11}[p])
        return dict({"kind": "assemble", "family": "nedelec", "degree": p}, **_ragged(rng, n),
                    assembly=rng.choice(["fp64", "fp64", "tf32x3"]) if p >= 3 else "fp64")
    if kind == "batch":
        large = rng.random() < 0.4
        lo = rng.randint(24, 60)
        return {"kind": "batch", "count": rng.randint(3, 6) if large else rng.randint(4, 20),
                "p1_min": 180 if large else lo,
                "p1_max": rng.randint(190, 400) if large else lo + rng.randint(10, 110),
                "p2_min": 17 if large else 6, "p2_max": rng.randint(18, 24) if large else 14,
                "mode": "cta_groups" if large else "cta_per_system"}
    p = rng.choice([1, 2, 3])
    n = _log_int(rng, 4, {1: 28, 2: 16, 3: 10}[p])
    return dict({"kind": rng.choice(["csc", "jvp", "vjp"]), "family": "lagrange", "degree": p},
                **_ragged(rng, n))


# ----------------------------------------------------------- sizes and work

def _sizes(case):
    """Cells, vertices, DoFs, free DoFs, stored entries and load points per cell."""
    f = case["family"]
    if f == "p1":
        nx, ny = case["nx"], case["ny"]
        free = (nx - 1) * (ny - 1)
        return 2 * nx * ny, (nx + 1) * (ny + 1), (nx + 1) * (ny + 1), free, 7 * free, 1
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells, verts, p = 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), case["degree"]
    if f == "lagrange":
        dofs = (p * nx + 1) * (p * ny + 1) * (p * nz + 1)
        free = (p * nx - 1) * (p * ny - 1) * (p * nz - 1)
        return cells, verts, dofs, free, int(free * {1: 15, 2: 29, 3: 50, 4: 77}[p]), _nq(f, p)
    edges = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
             + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
    bfaces = 4 * (nx * ny + ny * nz + nx * nz)
    faces = (4 * cells + bfaces) // 2
    dofs = edges * p + faces * p * (p - 1) + cells * (p * (p - 1) * (p - 2) // 2)
    free = dofs - bfaces * 3 // 2 * p - bfaces * p * (p - 1)
    return cells, verts, dofs, free, int(free * (4.5 * p + 6.5 * p * p + 4)), _nq(f, p)


def _nq(family, p):
    if p == 1 and family == "nedelec" or p <= 2 and family == "lagrange":
        return 4
    q = 2 * p + 2 if family == "nedelec" else 2 * p + 4
    return ((q + 4) // 2) ** 3


def work(case):
    """Inputs read once, outputs written once, and the operator's nonzeros (8
    bytes each) written once by the assembly; floating-point operations of the
    element matrices and of the CG iterations the solver's tolerance takes."""
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for s in _batch_systems(case):
            w = work(dict(s, kind="solve", precision="mixed"))
            total = {k: total[k] + w[k] for k in total}
        return total
    cells, verts, dofs, free, nnz, nq = _sizes(case)
    dim = 2 if case["family"] == "p1" else 3
    width = 3 if case["family"] == "nedelec" else 1
    nb = _nb(case)
    geometry = 8.0 * dim * verts + 4.0 * (dim + 1) * cells
    if case["kind"] in ("csc", "jvp", "vjp"):
        full = 8.0 * nnz * dofs / max(free, 1)
        return {"bytes": geometry + 1.5 * full, "flops": 14.0 * nb * nb * cells}
    inputs = geometry + 8.0 * cells + 8.0 * nq * width * cells
    contract = (24.0 if width == 3 else 14.0) * nb * nb * cells
    if case["kind"] == "assemble":
        return {"bytes": inputs + 8.0 * nnz + 32.0 * free, "flops": contract + 2.0 * nnz}
    n = max(case["nx"], case["ny"], case.get("nz", 0))
    its = {"p1": 4.5 * n, "lagrange": 7.0 * case.get("degree", 1) * n,
           "nedelec": 30.0 * case.get("degree", 1) ** 2 * n}[case["family"]]
    return {"bytes": inputs + 8.0 * nnz + 8.0 * dofs, "flops": contract + its * (2.0 * nnz + 10.0 * free)}


def _nb(case):
    p = case.get("degree", 1)
    return {"p1": 3, "lagrange": (p + 1) * (p + 2) * (p + 3) // 6,
            "nedelec": p * (p + 2) * (p + 3) // 2}[case["family"]]


def _batch_systems(case):
    """Two thirds P1 squares, one third P2 boxes, sizes spread over the case's ranges."""
    out, n = [], case["count"]
    for i in range(n):
        u = i / max(n - 1, 1)
        if i % 3 < 2:
            m = int(round(case["p1_min"] * (case["p1_max"] / case["p1_min"]) ** u))
            out.append({"family": "p1", "nx": m, "ny": m})
        else:
            m = int(round(case["p2_min"] * (case["p2_max"] / case["p2_min"]) ** u))
            out.append({"family": "lagrange", "degree": 2, "nx": m, "ny": m, "nz": m})
    return out


# ---------------------------------------------------------------- inputs

def _mesh(case):
    """Unjittered vertices (numpy, 3 or 2 columns) and cells."""
    if case["family"] != "p1":
        v, t, st = ff.generate_structured_tetra_box_mesh(
            [[0, 1], [0, 1], [0, 1]], [case["nx"], case["ny"], case["nz"]])
        if st.code:
            raise ValueError(st.message)
        return v, t
    nx, ny = case["nx"], case["ny"]
    x, y = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
    v = np.stack([x.ravel(), y.ravel()], 1)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    a = (j * (nx + 1) + i).ravel()
    b, c, d = a + 1, a + nx + 2, a + nx + 1
    t = np.stack([a, b, c, a, c, d], 1).reshape(-1, 3)
    return v, np.ascontiguousarray(t, dtype=np.int32)


def _gauss(m):
    x, w = np.polynomial.legendre.leggauss(m)
    return 0.5 * (x + 1.0), 0.5 * w


def _tet_rule(family, p, matrix=False):
    """Points (q, 3) and weights of the load rule (or of a rule exact for the matrix)."""
    if not matrix and _nq(family, p) == 4:
        a, b = (5.0 + 3.0 * 5.0 ** 0.5) / 20.0, (5.0 - 5.0 ** 0.5) / 20.0
        return np.array([[b, b, b], [a, b, b], [b, a, b], [b, b, a]]), np.full(4, 1.0 / 24.0)
    m = p + 2 if matrix else round(_nq(family, p) ** (1.0 / 3.0))
    t, w = _gauss(m)
    a, b, c = (g.ravel() for g in np.meshgrid(t, t, t, indexing="ij"))
    wa, wb, wc = (g.ravel() for g in np.meshgrid(w, w, w, indexing="ij"))
    pts = np.stack([a, (1 - a) * b, (1 - a) * (1 - b) * c], 1)
    return pts, wa * wb * wc * (1 - a) ** 2 * (1 - b)


def _inputs(case, seed):
    """Vertices, cells, cell coefficients and load samples, made on the GPU."""
    v0, t0 = _mesh(case)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    v, t = torch.as_tensor(v0, device=DEV), torch.as_tensor(t0, device=DEV).long()
    counts = torch.tensor([case["nx"], case["ny"], case.get("nz", 1)][:v.shape[1]], device=DEV)
    inner = ((v > 1e-9) & (v < 1 - 1e-9)).all(1, keepdim=True)
    jitter = (torch.rand(v.shape, generator=g, dtype=F64, device=DEV) - 0.5) * 0.2 / counts
    v = torch.where(inner, v + jitter, v).contiguous()
    width = 3 if case["family"] == "nedelec" else 1
    if width == 3:
        kappa = 0.5 + 1.5 * torch.rand(len(t), generator=g, dtype=F64, device=DEV)
    else:
        kappa = torch.exp(torch.randn(len(t), generator=g, dtype=F64, device=DEV))
    k = torch.randint(0, 3, (v.shape[1], 4), generator=g, device=DEV).double()
    ph = 2 * math.pi * torch.rand(4, generator=g, dtype=F64, device=DEV)
    amp = torch.randn(4, width, generator=g, dtype=F64, device=DEV)
    if case["family"] == "p1":
        x = v[t].mean(1, keepdim=True)
    else:
        xi = torch.as_tensor(_tet_rule(case["family"], case["degree"])[0], device=DEV)
        corners = v[t]
        x = corners[:, :1] + torch.einsum("qk,tkr->tqr", xi, corners[:, 1:] - corners[:, :1])
    samples = torch.cos(math.pi * (x @ k) + ph) @ amp
    return v, t, kappa, samples.contiguous(), g


_FAMILY = {"p1": ff.FFG_TRIANGLE_P1, "lagrange": ff.FFG_TETRA_LAGRANGE,
           "nedelec": ff.FFG_TETRA_NEDELEC}


def _mass(case):
    return 10.0 if case["family"] == "nedelec" else 0.0


def _problem(case, t, n_vertices):
    p = case.get("degree", 1)
    duffy = case["family"] == "lagrange" and p > 2
    return ff.Problem(_FAMILY[case["family"]], p, t.int().cpu().numpy(), n_vertices,
                      rule=ff.FFG_RULE_DUFFY if duffy else ff.FFG_RULE_DEGREE_TWO,
                      quadrature_degree=2 * p + 4 if duffy else 0, boundary="all")


def _options(case):
    return ff.SolverOptions(method="pcg", preconditioner="jacobi", tolerance=1e-10,
                            max_iterations=1000000, precision=case["precision"],
                            breakdown_guard="spd")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = [prepare(dict(s, kind="solve", precision="mixed", host=False), seed * 1009 + i)
                 for i, s in enumerate(_batch_systems(case))]
        return {"case": case, "parts": parts, "stream": torch.cuda.Stream(),
                "options": _options({"precision": "mixed"})}
    v, t, kappa, samples, g = _inputs(case, seed)
    s = {"case": case, "v": v, "t": t}
    if kind in ("csc", "jvp", "vjp"):
        s["v"], s["t"] = v.cpu().numpy(), t.int().cpu().numpy()
        if kind == "jvp":
            s["dot"] = torch.randn(v.shape, generator=g, dtype=F64, device=DEV).cpu().numpy()
        if kind == "vjp":
            A, st = ff.assemble_tetra_lagrange_stiffness_csc(s["v"], s["t"], case["degree"],
                                                             2 * case["degree"], 1.0, 0.5)
            assert st.code == 0, st.message
            s["bar"] = torch.randn(A.nnz, generator=g, dtype=F64, device=DEV).cpu().numpy()
        return s
    P = _problem(case, t, len(v))
    s.update(problem=P, kappa=kappa, samples=samples)
    if kind == "assemble":
        if case["assembly"] != "fp64":
            P.set_assembly_precision(case["assembly"])
        perm, st = np.zeros(P.n_free, np.int32), ctypes.c_int(0)
        K.load().ffg_problem_sell_permutation(P.handle, ctypes.c_void_p(perm.ctypes.data),
                                              ctypes.byref(st))
        assert st.value == 0
        perm = torch.as_tensor(perm, device=DEV).long()
        s["row_of_free"] = torch.empty_like(perm).scatter_(
            0, perm, torch.arange(P.n_free, device=DEV))
        x = torch.randn(P.n_free, generator=g, dtype=F64, device=DEV)
        s["x"] = x[perm].contiguous()
        s["out"] = [torch.zeros(P.n_free, dtype=F64, device=DEV) for _ in range(3)]
    elif case["host"]:
        s["options"] = _options(case)
        s["arrays"] = [a.cpu().numpy() for a in (v, kappa, samples)]
        s["out"] = np.zeros(P.n_dofs)
    else:
        s["options"] = _options(case)
        s["out"] = torch.zeros(P.n_dofs, dtype=F64, device=DEV)
    return s


# ------------------------------------------------------------------- a pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        P = s["problem"]
        if case["host"]:
            v, kappa, samples = s["arrays"]
            P.solve(v, 1.0, _mass(case), kappa, None, samples, None, s["options"], out=s["out"])
        else:
            P.solve_device(s["v"], s["out"], 1.0, _mass(case), s["kappa"], None, s["samples"],
                           None, s["options"])
        return {"solution": s["out"]}
    if kind == "assemble":
        return _run_assemble(s)
    if kind == "batch":
        parts, stream = s["parts"], s["stream"]
        stream.wait_stream(torch.cuda.current_stream())
        problems = [p["problem"] for p in parts]
        solve_batch(problems, [p["v"] for p in parts], [p["out"] for p in parts],
                    [1.0] * len(parts), [0.0] * len(parts), [p["kappa"] for p in parts], None,
                    [p["samples"] for p in parts], None, s["options"], case["mode"], stream)
        stream.synchronize()
        for p in problems:
            if not p.batch_stats().converged:
                raise RuntimeError("a system of the batch did not converge")
        return [p["out"] for p in parts]
    d = case["degree"]
    if kind == "csc":
        A, st = ff.assemble_tetra_lagrange_stiffness_csc(s["v"], s["t"], d, 2 * d, 1.0, 0.5)
    elif kind == "jvp":
        A, st = ff.assemble_tetra_lagrange_stiffness_csc_jvp(s["v"], s["t"], d, 2 * d, 1.0, 0.5,
                                                             s["dot"], 0.3, -0.2)
    else:
        vb, sb, mb, st = ff.assemble_tetra_lagrange_stiffness_csc_vjp(s["v"], s["t"], d, 2 * d,
                                                                      1.0, 0.5, s["bar"])
        return {"vertices_bar": vb, "coefficients_bar": np.array([sb, mb])}
    return {"col_ptr": A.col_ptr, "row_idx": A.row_idx, "val": A.val}


def _run_assemble(s):
    lib, P, st = K.load(), s["problem"], ctypes.c_int(0)
    rhs, dinv, y = s["out"]

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib.ffg_problem_assemble(P.handle, p(s["v"]), 1.0, _mass(s["case"]), p(s["kappa"]), None,
                             p(s["samples"]), None, 1, stream, ctypes.byref(st))
    if not st.value:
        lib.ffg_problem_system_arrays(P.handle, p(rhs), p(dinv), 1, stream, ctypes.byref(st))
    if not st.value:
        lib.ffg_problem_sell_spmv(P.handle, p(s["x"]), p(y), stream, ctypes.byref(st))
    if st.value:
        raise RuntimeError("assembly status %d" % st.value)
    rows = s["row_of_free"]
    return {"rhs": rhs[rows], "dinv": dinv[rows], "y": y[rows]}


# ------------------------------------------------------- the same in 64 bits

def _first_appearance(keys):
    """Ids of the keys (any shape) in order of first appearance."""
    _, first, inv = np.unique(keys.ravel(), return_index=True, return_inverse=True)
    rank = np.empty(len(first), np.int64)
    rank[np.argsort(first)] = np.arange(len(first))
    return rank[inv.ravel()].reshape(keys.shape)


def _lagrange_indices(p):
    return np.array([(a, b, c, p - a - b - c) for a in range(p + 1) for b in range(p + 1 - a)
                     for c in range(p + 1 - a - b)])


def _lagrange_basis(p, pts):
    """Values (q, nb) and reference gradients (q, nb, 3) of the nodal basis."""
    idx = _lagrange_indices(p)
    mono = [(a, b, c) for a in range(p + 1) for b in range(p + 1 - a) for c in range(p + 1 - a - b)]

    def table(x, d=None):
        cols = []
        for e in mono:
            f = 1.0
            e = list(e)
            if d is not None:
                f, e[d] = float(e[d]), max(e[d] - 1, 0)
            cols.append(f * x[:, 0] ** e[0] * x[:, 1] ** e[1] * x[:, 2] ** e[2])
        return np.stack(cols, 1)

    C = np.linalg.inv(table(idx[:, 1:] / p))
    return table(pts) @ C, np.stack([table(pts, d) @ C for d in range(3)], 2)


def _lagrange_elements(case, v, t, a, m):
    """Element matrices (T, nb, nb) with coefficients a (per cell) and m."""
    p = case["degree"]
    pts, w = _tet_rule("lagrange", p, matrix=True)
    val, grad = (torch.as_tensor(x, device=DEV) for x in _lagrange_basis(p, pts))
    w = torch.as_tensor(w, device=DEV)
    J = (v[t[:, 1:]] - v[t[:, :1]]).transpose(1, 2)
    Ji, det = torch.linalg.inv(J), torch.linalg.det(J)
    G = (a * det)[:, None, None] * (Ji @ Ji.transpose(1, 2))
    R = torch.einsum("q,qia,qjb->abij", w, grad, grad).reshape(9, -1)
    M = torch.einsum("q,qi,qj->ij", w, val, val)
    nb = val.shape[1]
    return (G.reshape(-1, 9) @ R).reshape(-1, nb, nb) + (m * det)[:, None, None] * M


def _lagrange_dofs(case, t):
    """Global DoFs (T, nb) and the boundary mask: DoFs are lattice points of the box."""
    n, p = [case["nx"], case["ny"], case["nz"]], case["degree"]
    t = t.cpu().numpy()
    ijk = np.stack([t % (n[0] + 1), t // (n[0] + 1) % (n[1] + 1), t // ((n[0] + 1) * (n[1] + 1))], 2)
    lat = np.einsum("bk,tkd->tbd", _lagrange_indices(p), ijk)
    key = lat[..., 0] + (p * n[0] + 1) * (lat[..., 1] + (p * n[1] + 1) * lat[..., 2])
    gd = _first_appearance(key)
    con = np.zeros(gd.max() + 1, bool)
    con[gd[((lat == 0) | (lat == p * np.array(n))).any(2)]] = True
    return torch.as_tensor(gd, device=DEV), torch.as_tensor(con, device=DEV)


def _jacobi_poly(n, alpha, x):
    """P_n^(alpha, 0) from its finite sum."""
    s = np.zeros_like(x)
    for k in range(n + 1):
        s = s + math.comb(n + alpha, n - k) * math.comb(n, k) * (0.5 * (x - 1)) ** k * (0.5 * (x + 1)) ** (n - k)
    return s


def _face_weight(k, a, b, u, v):
    if k <= 5:
        return u ** a * v ** b
    return _jacobi_poly(a, 0, 2 * u / (1 - v) - 1) * (1 - v) ** a * _jacobi_poly(b, 2 * a + 1, 2 * v - 1)


def _volume_weight(k, a, b, c, x):
    x, y, z = x.T
    if k <= 5:
        return x ** a * y ** b * z ** c
    return (_jacobi_poly(a, 0, 2 * x / (1 - y - z) - 1) * (1 - y - z) ** a
            * _jacobi_poly(b, 2 * a + 1, 2 * y / (1 - z) - 1) * (1 - z) ** b
            * _jacobi_poly(c, 2 * a + 2 * b + 2, 2 * z - 1))


def _nedelec_candidates(k, x):
    """Values and curls (q, nb, 3) of the first-kind space's monomial candidates."""
    d, terms = k - 1, []
    for comp in range(3):
        terms += [[(comp, 1.0, (a, b, e - a - b))] for e in range(k) for a in range(e + 1)
                  for b in range(e - a + 1)]
    for other in (1, 2):
        for a, b in ((a, b) for a in range(d + 1) for b in range(d - a + 1)):
            c = d - a - b
            lift = (a, b + 1, c) if other == 1 else (a, b, c + 1)
            terms.append([(0, -1.0, lift), (other, 1.0, (a + 1, b, c))])
    terms += [[(1, -1.0, (0, b, d - b + 1)), (2, 1.0, (0, b + 1, d - b))] for b in range(d + 1)]
    val, curl = np.zeros((len(x), len(terms), 3)), np.zeros((len(x), len(terms), 3))

    def mono(e):
        return x[:, 0] ** e[0] * x[:, 1] ** e[1] * x[:, 2] ** e[2]

    for i, term in enumerate(terms):
        for comp, s, e in term:
            val[:, i, comp] += s * mono(e)
            for ax in range(3):
                if ax != comp and e[ax]:
                    lower = list(e)
                    lower[ax] -= 1
                    # curl component: epsilon_{r, ax, comp}
                    r = 3 - ax - comp
                    sign = 1.0 if (ax, comp) in ((0, 1), (1, 2), (2, 0)) else -1.0
                    curl[:, i, r] += sign * s * e[ax] * mono(lower)
    return val, curl


_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
_FACES = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]


def _nedelec_basis(k, rank, x):
    """Values and curls at x of the basis dual to edge and face moments taken in
    the order `rank` of the cell's global vertices, and volume moments."""
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    t, w = _gauss(k + 2)
    rows = []
    for e in _EDGES:
        a, b = sorted(e, key=lambda i: rank[i])
        tan = V[b] - V[a]
        tr = _nedelec_candidates(k, V[a] + t[:, None] * tan)[0] @ tan
        rows += [(w * _jacobi_poly(m, 0, 2 * t - 1)) @ tr for m in range(k)]
    u, s = (g.ravel() for g in np.meshgrid(t, t, indexing="ij"))
    wu, ws = (g.ravel() for g in np.meshgrid(w, w, indexing="ij"))
    s, wf = (1 - u) * s, wu * ws * (1 - u)
    for f in _FACES:
        a, b, c = sorted(f, key=lambda i: rank[i])
        tans = V[b] - V[a], V[c] - V[a]
        val = _nedelec_candidates(k, V[a] + u[:, None] * tans[0] + s[:, None] * tans[1])[0]
        for tan in tans:
            rows += [(wf * _face_weight(k, ma, d - ma, u, s)) @ (val @ tan)
                     for d in range(k - 1) for ma in range(d + 1)]
    pts, wv = _tet_rule("nedelec", k + 1, matrix=True)
    val = _nedelec_candidates(k, pts)[0]
    for comp in range(3):
        rows += [(wv * _volume_weight(k, a, b, d - a - b, pts)) @ val[:, :, comp]
                 for d in range(k - 2) for a in range(d + 1) for b in range(d - a + 1)]
    C = np.linalg.inv(np.array(rows))
    val, curl = _nedelec_candidates(k, x)
    return np.einsum("qcr,cb->qbr", val, C), np.einsum("qcr,cb->qbr", curl, C)


def _nedelec_dofs(k, t):
    t = t.cpu().numpy().astype(np.int64)
    nv = t.max() + 1
    e = np.sort(t[:, _EDGES], 2)
    f = np.sort(t[:, _FACES], 2)
    fkey = (f[..., 0] * nv + f[..., 1]) * nv + f[..., 2]
    ei, fi = _first_appearance(e[..., 0] * nv + e[..., 1]), _first_appearance(fkey)
    fd, cd = k * (k - 1), k * (k - 1) * (k - 2) // 2
    ne, nf, T = ei.max() + 1, fi.max() + 1, len(t)
    gd = np.concatenate([
        (ei[:, :, None] * k + np.arange(k)).reshape(T, -1),
        (ne * k + fi[:, :, None] * fd + np.arange(fd)).reshape(T, -1),
        ne * k + nf * fd + np.arange(T)[:, None] * cd + np.arange(cd)], 1)
    con = np.zeros(ne * k + nf * fd + T * cd, bool)
    outer = (np.bincount(fi.ravel()) == 1)[fi]
    for lf, face in enumerate(_FACES):
        cells = np.nonzero(outer[:, lf])[0]
        con[gd[cells, 6 * k + lf * fd:6 * k + (lf + 1) * fd]] = True
        for pair in itertools.combinations(face, 2):
            le = _EDGES.index(pair)
            con[gd[cells, le * k:(le + 1) * k]] = True
    return torch.as_tensor(gd, device=DEV), torch.as_tensor(con, device=DEV)


def _nedelec_groups(k, t):
    """(cells, matrix basis, load basis, weights) of every vertex order among the cells."""
    ranks = torch.argsort(torch.argsort(t, 1), 1).cpu().numpy()
    kinds, of = np.unique(ranks, axis=0, return_inverse=True)
    mp, mw = _tet_rule("nedelec", k, matrix=True)
    lp, lw = _tet_rule("nedelec", k)
    for i, r in enumerate(kinds):
        up = [torch.as_tensor(x, device=DEV) for x in (*_nedelec_basis(k, r, mp), mw,
                                                      _nedelec_basis(k, r, lp)[0], lw)]
        cells = torch.as_tensor(np.nonzero(of.ravel() == i)[0], device=DEV)
        for part in cells.split(4096):
            yield part, up


def _geometry(v, t):
    J = (v[t[:, 1:]] - v[t[:, :1]]).transpose(1, 2)
    return J, torch.linalg.inv(J), torch.linalg.det(J)


def _exact_nedelec(case, seed):
    v, t, mu, samples, g = _inputs(case, seed)
    k, mass = case["degree"], _mass(case)
    gd, con = _nedelec_dofs(k, t)
    free = torch.nonzero(~con).ravel()
    n = len(con)
    rhs = torch.zeros(n, dtype=F64, device=DEV)
    diag, y, x = torch.zeros_like(rhs), torch.zeros_like(rhs), torch.zeros_like(rhs)
    solve = case["kind"] == "solve"
    if not solve:
        x[free] = torch.randn(len(free), generator=g, dtype=F64, device=DEV)
    elements = torch.empty(len(t), gd.shape[1], gd.shape[1], dtype=F64, device=DEV) if solve else None
    for c, (val, curl, w, lval, lw) in _nedelec_groups(k, t):
        J, Ji, det = _geometry(v, t[c])
        cw = (mu[c] / det)[:, None, None] * (J.transpose(1, 2) @ J)
        mw = (mass * det)[:, None, None] * (Ji @ Ji.transpose(1, 2))
        f = det[:, None, None] * torch.einsum("tab,tqb->tqa", Ji, samples[c])
        F = torch.einsum("q,tqa,qia->ti", lw, f, lval)
        rhs.index_add_(0, gd[c].ravel(), F.ravel())
        if solve:
            for B, W in ((curl, cw), (val, mw)):
                R = torch.einsum("q,qia,qjb->abij", w, B, B).reshape(9, -1)
                part = (W.reshape(-1, 9) @ R).reshape(len(c), *elements.shape[1:])
                elements[c] = part if B is curl else elements[c] + part
            continue
        out = 0.0
        dg = 0.0
        for B, W in ((curl, cw), (val, mw)):
            u = (x[gd[c]] @ B.transpose(0, 1).reshape(B.shape[1], -1)).reshape(len(c), -1, 3)
            u = torch.einsum("q,tab,tqb->tqa", w, W, u).reshape(len(c), -1)
            out = out + u @ B.transpose(0, 1).reshape(B.shape[1], -1).T
            dg = dg + W.reshape(-1, 9) @ torch.einsum("q,qia,qib->abi", w, B, B).reshape(9, -1)
        y.index_add_(0, gd[c].ravel(), out.ravel())
        diag.index_add_(0, gd[c].ravel(), dg.ravel())
    if solve:
        return {"solution": _cg(elements, gd, con, rhs)}
    return {"rhs": rhs[free], "dinv": 1.0 / diag[free], "y": y[free]}


def _cg(elements, gd, con, rhs):
    """Solution over all DoFs, zero where constrained: Jacobi-CG until the residual
    has fallen by 1e-14."""
    n = len(con)
    i = gd[:, :, None].expand_as(elements).reshape(-1)
    j = gd[:, None, :].expand_as(elements).reshape(-1)
    keep = ~con[i] & ~con[j]
    A = torch.sparse_coo_tensor(torch.stack([i[keep], j[keep]]), elements.reshape(-1)[keep],
                                (n, n)).coalesce()
    ij, a = A.indices(), A.values()
    d = torch.ones(n, dtype=F64, device=DEV)
    on = ij[0] == ij[1]
    d[ij[0][on]] = a[on]
    A = A.to_sparse_csr()
    b = torch.where(con, torch.zeros_like(rhs), rhs)
    x, best = torch.zeros_like(b), float("inf")
    for _ in range(4):  # restarted from the true residual
        r = b - A @ x
        if not float(r.norm()) < 0.5 * best or float(r.norm()) == 0.0:
            break
        best = float(r.norm())
        z = r / d
        p, rz, step, first = z.clone(), r @ z, 0, float(r.norm())
        while step < 20000:
            for _ in range(50):
                q = A @ p
                alpha = rz / (p @ q)
                x, r = x + alpha * p, r - alpha * q
                z = r / d
                new = r @ z
                p, rz = z + (new / rz) * p, new
            step += 50
            if not float(r.norm()) > 1e-14 * first:
                break
    return x


def _exact_scalar(case, seed):
    v, t, kappa, samples, _ = _inputs(case, seed)
    if case["family"] == "p1":
        x, y = v[t][..., 0], v[t][..., 1]
        det = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
        gx = torch.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], 1) / det[:, None]
        gy = torch.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], 1) / det[:, None]
        area = 0.5 * det.abs()
        E = (kappa * area)[:, None, None] * (gx[:, :, None] * gx[:, None] + gy[:, :, None] * gy[:, None])
        F = (samples.reshape(-1) * area / 3.0)[:, None].expand(-1, 3)
        i, j = np.meshgrid(np.arange(case["nx"] + 1), np.arange(case["ny"] + 1))
        con = (i == 0) | (i == case["nx"]) | (j == 0) | (j == case["ny"])
        gd, con = t, torch.as_tensor(con.ravel(), device=DEV)
    else:
        one = torch.ones_like(kappa)
        E = _lagrange_elements(case, v, t, kappa, 0.0 * one)
        gd, con = _lagrange_dofs(case, t)
        pts, w = _tet_rule("lagrange", case["degree"])
        B = torch.as_tensor(w[:, None] * _lagrange_basis(case["degree"], pts)[0], device=DEV)
        F = _geometry(v, t)[2][:, None] * (samples[..., 0] @ B)
    rhs = torch.zeros(len(con), dtype=F64, device=DEV).index_add_(0, gd.reshape(-1), F.reshape(-1))
    return {"solution": _cg(E, gd, con, rhs)}


def _exact_csc(case, seed):
    v, t, _, _, g = _inputs(case, seed)
    gd, con = _lagrange_dofs(case, t)
    n, nb = len(con), gd.shape[1]
    key = gd[:, None, :] * n + gd[:, :, None]  # column-major: column j, row i
    keys, at = torch.unique(key.reshape(-1), return_inverse=True)
    one = torch.ones(len(t), dtype=F64, device=DEV)

    def values(v, a, m):
        E = _lagrange_elements(case, v, t, a * one, m * one)
        return torch.zeros(len(keys), dtype=F64, device=DEV).index_add(0, at, E.reshape(-1))

    a = torch.tensor(1.0, dtype=F64, device=DEV)
    m = torch.tensor(0.5, dtype=F64, device=DEV)
    if case["kind"] == "vjp":
        bar = torch.randn(len(keys), generator=g, dtype=F64, device=DEV)
        args = [x.clone().requires_grad_(True) for x in (v, a, m)]
        grads = torch.autograd.grad((values(*args) * bar).sum(), args)
        return {"vertices_bar": grads[0], "coefficients_bar": torch.stack(grads[1:])}
    col_ptr = torch.searchsorted(keys, torch.arange(n + 1, device=DEV) * n)
    val = values(v, a, m)
    if case["kind"] == "jvp":
        dot = torch.randn(v.shape, generator=g, dtype=F64, device=DEV)
        da, dm = torch.full_like(a, 0.3), torch.full_like(m, -0.2)
        val = torch.func.jvp(values, (v, a, m), (dot, da, dm))[1]
    return {"col_ptr": col_ptr, "row_idx": (keys % n).int(), "val": val}


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_scalar(dict(s, kind="solve"), seed * 1009 + i)["solution"]
                for i, s in enumerate(_batch_systems(case))]
    if case["kind"] in ("csc", "jvp", "vjp"):
        return _exact_csc(case, seed)
    return _exact_nedelec(case, seed) if case["family"] == "nedelec" else _exact_scalar(case, seed)
