"""Host threads that run the same kernels at different sizes at the same time:
every call succeeds and returns what it returns alone."""
import threading

import numpy as np
import pytest

import oracle
import fortfem_b200 as ff
from fortfem_b200 import _capi as K

pytestmark = pytest.mark.gpu


def together(calls, repeats):
    """Each call's results alone, then `repeats` of all calls in threads of their own."""
    want = [c() for c in calls]
    wrong = []
    start = threading.Barrier(len(calls))

    def loop(call, expected):
        start.wait()
        for _ in range(repeats):
            try:
                if not np.array_equal(call(), expected):
                    wrong.append("other values")
            except Exception as e:  # the library's error, reported by the test's thread
                wrong.append(str(e))

    threads = [threading.Thread(target=loop, args=(c, w)) for c, w in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[0])


def test_assemblies_of_meshes_with_different_columns():
    """A fan of 400 triangles (a column of 401 entries) beside a regular square."""
    n = 400
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    fan_v = np.vstack([[0.0, 0.0], np.stack([np.cos(a), np.sin(a)], -1)])
    i = np.arange(n)
    fan_t = np.stack([np.zeros(n, int), 1 + i, 1 + (i + 1) % n], -1).astype(np.int32)
    sq_v, sq_t = oracle.unit_square_mesh(30)

    def solver(v, t, boundary):
        prob = ff.Problem(K.FFG_TRIANGLE_P1, 1, t, len(v), boundary=boundary)
        src = np.ones(prob.sample_points(v).shape[:-1])
        opts = ff.SolverOptions(method="pcg", preconditioner="jacobi", tolerance=1e-10,
                                precision="mixed")
        return lambda: prob.solve(v, 1.0, 1.0, None, None, src, None, opts)[0]

    together([solver(fan_v, fan_t, "none"), solver(sq_v, sq_t, "none")], 100)


def test_adjoints_of_different_orders():
    """Nedelec adjoints of orders 5 (182 KB of shared memory) and 6 (59 KB)."""
    v, t = oracle.box_mesh([1, 1, 1])

    def adjoint(order):
        A, st = ff.assemble_tetra_nedelec_curl_mass_csc(v, t, order=order)
        assert st.code == 0, st.message
        bar = np.random.default_rng(order).standard_normal(len(A.val))

        def call():
            out = ff.assemble_tetra_nedelec_curl_mass_csc_vjp(v, t, order, 1.0, 1.0, bar)
            assert out[-1].code == 0, out[-1].message
            return out[0]
        return call

    together([adjoint(5), adjoint(6)], 40)
