"""The solver's operator as the slice gathers assemble it: rows, diagonal and
right-hand side (with Dirichlet lifting) against the FP64 CPU oracle.

Tolerances are those of the CSC parity tests (relative Frobenius 1e-12; 1e-11
and 1e-10 at Nedelec orders 5 and 6, whose tables carry larger entries), the
matrix through A x for a random x, so relative to | |A| |x| |.
"""
import ctypes

import numpy as np
import pytest

import oracle
import fortfem_b200 as ff
from fortfem_b200 import _capi as K
from fortfem_b200 import synth
from fortfem_b200.api import solve_batch

pytestmark = pytest.mark.gpu


def fan(n):
    """n tetrahedra around one edge: an edge (and, for Lagrange elements, two
    vertices) with n incidences and a row as long as the mesh has DoFs."""
    a = 2 * np.pi * np.arange(n) / n
    r = 1.0 + 0.1 * np.cos(3 * a)
    v = np.concatenate([[[0.0, 0.0, -0.5], [0.1, 0.05, 0.6]],
                        np.stack([r * np.cos(a), r * np.sin(a), 0.1 * np.sin(2 * a)], -1)])
    i = np.arange(n)
    t = np.stack([0 * i, 0 * i + 1, 2 + i, 2 + (i + 1) % n], -1).astype(np.int32)
    d = v[t[:, 1:]] - v[t[:, :1]]
    assert (np.linalg.det(d) > 0).all()
    return v, t


def box(n):
    v, t = oracle.box_mesh([n, n, n])
    return synth.jitter_interior(v, 1.0 / n, 0.1, 5), t


def operator(prob, v, ca, cb, cell_a, src, g, x, assemble=True):
    """rhs, 1 / diagonal and A x, in the order of the free DoFs."""
    import torch

    def p(a):
        return ctypes.c_void_p(a.data_ptr())

    dev = [torch.as_tensor(a, device="cuda") for a in (v, cell_a, src, g)]
    perm, st = np.zeros(prob.n_free, np.int32), ctypes.c_int(0)
    lib = K.load()
    lib.ffg_problem_sell_permutation(prob.handle, ctypes.c_void_p(perm.ctypes.data),
                                     ctypes.byref(st))
    assert st.value == 0
    xs = torch.as_tensor(x[perm], device="cuda")
    rhs, dinv, y = (torch.zeros(prob.n_free, dtype=torch.float64, device="cuda") for _ in range(3))
    if assemble:
        lib.ffg_problem_assemble(prob.handle, p(dev[0]), ca, cb, p(dev[1]), None, p(dev[2]),
                                 p(dev[3]), 1, None, ctypes.byref(st))
    assert st.value == 0
    lib.ffg_problem_system_arrays(prob.handle, p(rhs), p(dinv), 1, None, ctypes.byref(st))
    assert st.value == 0
    lib.ffg_problem_sell_spmv(prob.handle, p(xs), p(y), None, ctypes.byref(st))
    assert st.value == 0
    torch.cuda.synchronize()
    out = []
    for a in (rhs, dinv, y):
        b = np.zeros(prob.n_free)
        b[perm] = a.cpu().numpy()
        out.append(b)
    return out


NEDELEC = [  # 8 lanes per row at order 1, 16 per row, 32 where the order or a long row asks for it
    (1, "box", 2), (2, "box", 2), (3, "box", 2), (4, "box", 2), (5, "box", 1), (6, "box", 1),
    (1, "fan", 40),
    (2, "fan", 24), (2, "fan", 70), (3, "fan", 40), (4, "fan", 20), (4, "fan", 60), (5, "fan", 9),
]


@pytest.mark.parametrize("k, mesh, n", NEDELEC)
def test_nedelec_rows_match_oracle(k, mesh, n):
    v, t = box(n) if mesh == "box" else fan(n)
    rng = np.random.default_rng(10 * k + n)
    n_dofs = oracle.nedelec_csc(v, t, k, 1.0, 1.0)[0] if k < 6 else 1014
    mask = rng.random(n_dofs) < 0.15
    cell = rng.uniform(0.5, 2.0, len(t))
    pts = oracle.nedelec_load_points(v, t, k)
    src = np.stack([np.sin(pts[..., 1]), pts[..., 0] * pts[..., 2], np.cos(pts[..., 0])], -1)
    g = np.where(mask, rng.standard_normal(n_dofs), 0.0)
    check(ff.Problem(K.FFG_TETRA_NEDELEC, k, t, len(v), boundary=mask.astype(np.uint8)), v, 1.7,
          0.9, cell, src, g, mask, oracle.nedelec_csc(v, t, k, 1.7, 0.9, cell, None),
          oracle.nedelec_load_samples(v, t, k, src), {5: 1e-11, 6: 1e-10}.get(k, 1e-12), rng)


LAGRANGE = [  # 4 lanes per row (p = 1), 8, 16 where a long row asks for it, a thread
    (1, "box", 2), (2, "box", 2), (3, "box", 2), (4, "box", 1), (1, "fan", 70), (2, "fan", 60),
    (2, "fan", 90), (3, "fan", 40), (4, "fan", 20), (4, "fan", 100),
]


def lagrange_case(p, mesh, n):
    v, t = box(n) if mesh == "box" else fan(n)
    q = p + 2
    rng = np.random.default_rng(10 * p + n)
    n_dofs = oracle.lagrange_csc(v, t, p, 0, q)[0]
    mask = rng.random(n_dofs) < 0.15
    cell = rng.uniform(0.5, 2.0, len(t))
    pts = oracle.lagrange_quadrature_points(v, t, 0, q)
    src = np.sin(pts[..., 0]) * np.cos(2 * pts[..., 1]) + pts[..., 2]
    g = np.where(mask, rng.standard_normal(n_dofs), 0.0)
    prob = ff.Problem(K.FFG_TETRA_LAGRANGE, p, t, len(v), quadrature_degree=q,
                      boundary=mask.astype(np.uint8))
    return prob, v, t, q, cell, src, g, mask, rng


@pytest.mark.parametrize("p, mesh, n", LAGRANGE)
def test_lagrange_rows_match_oracle(p, mesh, n):
    prob, v, t, q, cell, src, g, mask, rng = lagrange_case(p, mesh, n)
    check(prob, v, 1.7, 0.9, cell, src, g, mask, oracle.lagrange_csc(v, t, p, 0, q, 1.7, 0.9, cell),
          oracle.lagrange_load_samples(v, t, p, src, 0, q), 1e-12, rng)


@pytest.mark.parametrize("n", [3, 40])
def test_p1_triangle_rows_match_oracle(n):
    if n == 3:
        v, t = oracle.unit_square_mesh(n + 1)
    else:  # n triangles around one vertex
        a = 2 * np.pi * np.arange(n) / n
        v = np.concatenate([[[0.1, 0.0]], np.stack([np.cos(a), np.sin(a)], -1)])
        i = np.arange(n)
        t = np.stack([0 * i, 1 + i, 1 + (i + 1) % n], -1).astype(np.int32)
    rng = np.random.default_rng(n)
    mask = rng.random(len(v)) < 0.15
    mask[0] = False
    cell = rng.uniform(0.5, 2.0, len(t))
    g = np.where(mask, rng.standard_normal(len(v)), 0.0)
    check(ff.Problem(K.FFG_TRIANGLE_P1, 1, t, len(v), boundary=mask.astype(np.uint8)), v, 1.7, 0.9,
          cell, np.ones(len(t)), g, mask, oracle.p1_csc(v, t, 0.9, 1.7, cell),
          oracle.p1_load(v, t), 1e-12, rng)


def test_batched_rows_are_the_bits_of_a_system_alone():
    import torch

    cases = [lagrange_case(*c) for c in [(2, "box", 2), (1, "box", 2), (3, "fan", 40),
                                         (2, "fan", 90), (2, "fan", 60)]]
    for i, _ in enumerate(cases):
        rng = np.random.default_rng(i)
        prob, v, t, q, cell, src, g, mask, _ = cases[i]
        x = rng.standard_normal(prob.n_free)
        cases[i] = (prob, v, cell, src, g, x, operator(prob, v, 1.7, 0.9, cell, src, g, x))
    probs = [c[0] for c in cases]
    dev = [[torch.as_tensor(c[k], device="cuda") for c in cases] for k in (1, 2, 3, 4)]
    sol = [torch.zeros(p.n_dofs, dtype=torch.float64, device="cuda") for p in probs]
    solve_batch(probs, dev[0], sol, [1.7] * 5, [0.9] * 5, dev[1], None, dev[2], dev[3])
    torch.cuda.synchronize()
    for prob, v, cell, src, g, x, alone in cases:
        for a, b in zip(alone, operator(prob, v, 1.7, 0.9, cell, src, g, x, assemble=False)):
            assert np.array_equal(a, b)
        prob.close()


def check(problem, v, ca, cb, cell, src, g, mask, csc, load, tol, rng):
    nf, cp, ri, val, b, free = oracle.reduce_constrained(*csc, load, mask, g)
    A = oracle.csc_to_scipy(nf, cp, ri, val)
    x = rng.standard_normal(nf)
    with problem:
        assert problem.n_free == nf
        rhs, dinv, y = operator(problem, v, ca, cb, cell, np.ascontiguousarray(src), g, x)
    size = np.linalg.norm
    lifted = abs(oracle.csc_to_scipy(*csc)) @ abs(g)
    assert size(y - A @ x) <= tol * size(abs(A) @ abs(x))
    assert size(1.0 / dinv - A.diagonal()) <= tol * size(val)
    assert size(rhs - b) <= tol * (size(load) + size(lifted))


@pytest.mark.parametrize("nedelec", [False, True])
def test_csc_in_one_call_is_the_csc_by_size(nedelec, monkeypatch):
    from fortfem_b200 import api

    v, t = box(2)
    def call():
        if nedelec:
            return ff.assemble_tetra_nedelec_curl_mass_csc(v, t, 1.7, 0.9, order=2)
        return ff.assemble_tetra_lagrange_stiffness_csc(v, t, 3, 5, 1.7, 0.9)
    one, st = call()
    assert st.code == 0
    monkeypatch.setattr(api, "_CSC_BOUND_BYTES", 0)
    two, st = call()
    assert st.code == 0 and one.nrow == two.nrow and one.ncol == two.ncol
    for a in ("col_ptr", "row_idx", "val"):
        assert np.array_equal(getattr(one, a), getattr(two, a))
