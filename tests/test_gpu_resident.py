"""The on-chip PCG kernels (a cluster per system, the whole grid with the
operator in shared memory) at the edges of their partitions: fewer slices than
CTAs, partial last slices, rows long enough to be split, int32 columns,
operators larger than shared memory; FP64 and mixed.

The systems are strictly diagonally dominant, |a_ii| >= 2 sum |a_ij|, so
the Jacobi-scaled operator has its spectrum in [1/2, 3/2] and the solution's
relative error (in the scaled norm) is at most 3 times the relative residual;
the row scales spread over a factor 4, hence 12 tol = 1.2e-9 below.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import fortfem_b200 as ff
from fortfem_b200 import _capi as K

pytestmark = pytest.mark.gpu
TOL = 1e-10


def dominant(n, per_row, span, seed, long_rows=0):
    """Symmetric, 2 x diagonally dominant, about per_row entries a row within `span`."""
    rng = np.random.default_rng(seed)
    m = n * max(per_row - 1, 0) // 2
    i = rng.integers(0, n, m)
    j = np.clip(i + rng.integers(-span, span + 1, m), 0, n - 1)
    if long_rows:
        rows = rng.choice(n, long_rows, replace=False)
        i = np.concatenate([i] + [np.full(min(n, 300), r) for r in rows])
        j = np.concatenate([j] + [rng.choice(n, min(n, 300), replace=False) for _ in rows])
    v = rng.standard_normal(len(i))
    keep = i != j
    A = sp.coo_matrix((v[keep], (i[keep], j[keep])), shape=(n, n)).tocsr()
    A = A + A.T
    d = np.maximum(2.0 * np.asarray(abs(A).sum(axis=1)).ravel(), 1.0) * rng.uniform(1.0, 4.0, n)
    return (A + sp.diags(d)).tocsc()


def solve(A, b, precision):
    A.sort_indices()
    M = ff.CscMatrix(*A.shape, A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data)
    x = np.zeros(len(b))
    st = ff.solve_sparse(M, b, x, ff.solver_options(
        method="pcg", preconditioner="jacobi", tolerance=TOL, precision=precision,
        max_iterations=10000, breakdown_guard="spd"))
    return x, st


CASES = [
    # rows, entries a row, span, rows of 300 entries
    (1, 1, 1, 0), (2, 2, 1, 0), (31, 5, 30, 0), (33, 5, 32, 0), (257, 7, 40, 0),
    (511, 300, 510, 0),       # 16 slices, every one split into parts
    (513, 7, 512, 3),         # 17 slices over 16 CTAs, a few long rows
    (4097, 9, 4000, 5),       # two sigma windows
    (12001, 25, 12000, 4),    # cluster (mixed) or grid (FP64)
    (30011, 7, 180, 0),       # banded: the cluster exchanges its borders only
    (40009, 12, 40000, 2),    # grid, int32 columns
    (70001, 60, 3000, 0),     # grid, part of the operator left in L2
    (260003, 5, 500, 0),      # grid, many rows a CTA
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,per_row,span,long_rows", CASES)
def test_resident_solve_matches_direct(n, per_row, span, long_rows, precision):
    A = dominant(n, per_row, span, n, long_rows)
    xs = np.random.default_rng(n + 1).standard_normal(n)
    b = A @ xs
    x, st = solve(A, b, precision)
    assert st.converged and st.true_relative_residual <= 1.01 * TOL
    assert np.linalg.norm(x - xs) <= 12 * TOL * np.linalg.norm(xs)
    # the same bits again
    y, _ = solve(A, b, precision)
    assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_resident_hard_system_falls_back_like_the_staged_kernel(precision):
    """cond ~ 1e11: the mixed loop leaves FP32 (direct form, FP64 continuation) and
    both precisions end on the true residual they report."""
    n = 600
    A = sp.diags([np.full(n - 1, -1.0), np.full(n, 2.0), np.full(n - 1, -1.0)], [-1, 0, 1])
    A = (A @ A + 1e-9 * sp.identity(n)).tocsc()
    b = np.ones(n)
    x, st = solve(A, b, precision)
    res = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    assert np.isfinite(x).all()
    # FP64 rounding of one evaluation of b - A x
    floor = 1e-16 * np.linalg.norm(np.abs(A) @ np.abs(x)) / np.linalg.norm(b)
    assert abs(res - st.true_relative_residual) <= 1e-3 * res + 20 * floor


@pytest.mark.parametrize("n", [5, 40, 479, 4096, 6001])
@pytest.mark.parametrize("block", [1, 4])
def test_cluster_fp64_without_coupling_between_ctas(n, block):
    """Operators of which no CTA reads another's rows: the FP64 loop's exchange
    then copies nothing and is only held together by its messages.  Blocks of 4
    consecutive rows, so equal rows keep a slice's blocks together."""
    rng = np.random.default_rng(n + block)
    blocks = []
    for k in range(0, n, block):
        m = min(block, n - k)
        a = rng.uniform(-1.0, 1.0, (m, m))
        a = np.triu(a, 1) + np.triu(a, 1).T
        blocks.append(a + np.diag(2.0 * abs(a).sum(axis=1) + rng.uniform(1.0, 4.0, m)))
    A = sp.block_diag([sp.coo_matrix(k) for k in blocks]).tocsc()
    xs = rng.standard_normal(n)
    b = A @ xs
    x, st = solve(A, b, "fp64")
    assert st.converged and st.true_relative_residual <= 1.01 * TOL
    # |A^-1| <= 1 (diagonal less the rest of the row), |A| <= 13 (diagonal at most
    # 2 * 3 + 4, the rest 3)
    assert np.linalg.norm(x - xs) <= 1.01 * 13 * TOL * np.linalg.norm(xs)
    y, _ = solve(A, b, "fp64")
    assert np.array_equal(x, y)


def _hard(family, n, relabel):
    """A problem whose mixed solve stagnates, its inputs and options: P1 on n^2
    vertices with log-normal coefficients to the end of FP64's reach, or order-1
    Nedelec with a small mass."""
    rng = np.random.default_rng(n)
    if family == K.FFG_TRIANGLE_P1:
        v, t = oracle.unit_square_mesh(n)
        if relabel:
            new = rng.permutation(len(v))
            w = np.empty_like(v)
            w[new] = v
            v, t = w, new[t].astype(t.dtype)
        prob = ff.Problem(family, 1, t, len(v))
        inputs = (v, 1.0, 0.0, np.exp(rng.standard_normal(len(t))), None,
                  np.sin(3 * prob.sample_points(v)[..., 0]), None)
        tol = 1e-13
    else:
        v, t = oracle.box_mesh([n, n, n])
        prob = ff.Problem(family, 1, t, len(v))
        p = prob.sample_points(v)
        inputs = (v, 1.0, 1e-4, None, None,
                  np.stack([np.sin(3 * p[..., 1]), np.cos(p[..., 2]), p[..., 0]], -1), None)
        tol = 1e-10
    return prob, inputs, ff.SolverOptions(method="pcg", preconditioner="jacobi", tolerance=tol,
                                          precision="mixed", max_iterations=200000,
                                          breakdown_guard="spd")


@pytest.mark.parametrize("family,n,relabel", [
    (K.FFG_TETRA_NEDELEC, 8, False),    # both replicas fit a CTA
    (K.FFG_TETRA_NEDELEC, 16, False),   # FP64's published vector in global memory
    (K.FFG_TRIANGLE_P1, 160, False),    # the same, 16-bit column differences
    (K.FFG_TRIANGLE_P1, 190, True),     # the same, int32 columns
])
def test_cluster_mixed_solve_continues_in_fp64(family, n, relabel):
    """Direct form, reliable updates and the FP64 continuation of the cluster
    kernel: the continuation runs, the reported residual is the solution's, and it
    meets the tolerance or what FP64 can tell from zero.  Error of b - A x in FP64
    with m terms a row: (m + 1) u (|A| |x| + |b|); a solve ends when an update of x
    no longer halves the residual, so at no more than about twice that and the
    rounding of x itself, u |A| |x|."""
    prob, inputs, opts = _hard(family, n, relabel)
    with prob:
        sol, st = prob.solve(*inputs, opts)
        assert prob.phase_times()["fp64_continuation"]
        again, st2 = prob.solve(*inputs, opts)
        assert np.array_equal(sol, again) and st.iterations == st2.iterations
        A, rhs, free = prob.reduced_system(*inputs)[:3]
    M = sp.csc_matrix((A.val, A.row_idx, A.col_ptr), shape=(len(rhs), len(rhs)))
    x = sol[free]
    norm = np.linalg.norm(rhs)
    terms = np.diff(M.indptr).max()
    level = 1.2e-16 * np.linalg.norm(abs(M) @ abs(x) + abs(rhs)) / norm
    res = np.linalg.norm(rhs - M @ x) / norm
    assert abs(res - st.true_relative_residual) <= 2 * (terms + 1) * level
    assert st.converged or family == K.FFG_TRIANGLE_P1
    assert res <= max(1.01 * opts.tolerance, 2 * (terms + 2) * level)


@pytest.mark.parametrize("precision,n,per_row,span", [
    ("mixed", 257, 7, 40), ("fp64", 257, 7, 40),                  # cluster
    ("mixed", 40009, 12, 40000), ("fp64", 40009, 12, 40000),      # grid
    ("mixed16", 4097, 9, 4000), ("fp64", 900001, 12, 30000),      # streamed
])
def test_wall_limit_is_looked_at_every_iteration(precision, n, per_row, span):
    """Solves of some tens of iterations, with a limit that has passed at the first."""
    A = dominant(n, per_row, span, n)
    b = np.random.default_rng(n).standard_normal(n)
    A.sort_indices()
    M = ff.CscMatrix(n, n, A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data)
    opts = ff.solver_options(method="pcg", preconditioner="jacobi", tolerance=TOL,
                             precision=precision, max_iterations=60, breakdown_guard="spd")
    st = ff.solve_sparse(M, b, np.zeros(n), opts)
    assert st.converged and 5 < st.iterations < 60
    opts.timeout_seconds = 1e-9
    with pytest.raises(ff.FortfemError) as e:
        ff.solve_sparse(M, b, np.zeros(n), opts)
    assert e.value.code == K.FFG_TIMEOUT


@pytest.mark.parametrize("mode", ["cta_per_system", "cta_groups", "whole_device"])
@pytest.mark.parametrize("precision", ["mixed", "mixed16"])
def test_wall_limit_of_a_batch(mode, precision):
    import torch
    from fortfem_b200.api import solve_batch
    probs, inputs = [], []
    for k, n in enumerate((9, 14)):
        v, t = oracle.unit_square_mesh(n)
        probs.append(ff.Problem(K.FFG_TRIANGLE_P1, 1, t, len(v)))
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        src = np.ones(probs[-1].sample_points(v).shape[:-1])
        inputs.append((dev(v), dev(src)))
    for limit, want in ((1e-9, False), (60.0, True)):
        opts = ff.SolverOptions(method="pcg", preconditioner="jacobi", tolerance=TOL,
                                precision=precision, timeout_seconds=limit)
        out = [torch.empty(p.n_dofs, dtype=torch.float64, device="cuda") for p in probs]
        solve_batch(probs, [i[0] for i in inputs], out, [1.0, 1.0], [0.0, 0.0],
                    samples=[i[1] for i in inputs], options=opts, mode=mode)
        torch.cuda.synchronize()
        for p in probs:
            if want:
                assert p.batch_stats().converged
            else:
                with pytest.raises(ff.FortfemError) as e:
                    p.batch_stats()
                assert e.value.code == K.FFG_TIMEOUT
    for p in probs:
        p.close()


def test_half_precision_groups_match_alone():
    """MIXED16 systems side by side, each the bits of its own launch and, as a
    solution, within the residual of the whole device's."""
    import torch
    from fortfem_b200.api import solve_batch
    probs, vs, fs = [], [], []
    for n in (20, 45, 90, 140):
        v, t = oracle.unit_square_mesh(n)
        probs.append(ff.Problem(K.FFG_TRIANGLE_P1, 1, t, len(v)))
        vs.append(torch.from_numpy(np.ascontiguousarray(v)).cuda())
        fs.append(torch.ones(probs[-1].sample_points(v).shape[:-1], dtype=torch.float64,
                             device="cuda"))
    opts = ff.SolverOptions(method="pcg", preconditioner="jacobi", tolerance=TOL,
                            precision="mixed16", max_iterations=1000000)

    def run(which, mode):
        out = [torch.empty(probs[i].n_dofs, dtype=torch.float64, device="cuda") for i in which]
        one = [1.0] * len(which)
        solve_batch([probs[i] for i in which], [vs[i] for i in which], out, one, one,
                    samples=[fs[i] for i in which], options=opts, mode=mode)
        torch.cuda.synchronize()
        for i in which:
            st = probs[i].batch_stats()
            assert st.converged and st.true_relative_residual <= 1.01 * TOL
        return [o.cpu().numpy() for o in out]

    together = run(range(4), "cta_groups")
    for i in range(4):
        assert np.array_equal(run([i], "cta_groups")[0], together[i])
        whole = run([i], "whole_device")[0]
        assert np.linalg.norm(whole - together[i]) <= 1e-6 * np.linalg.norm(whole)
    for p in probs:
        p.close()
