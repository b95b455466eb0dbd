"""Stored Lanczos vectors that a build did not write take no part in its apply:
where every column stops early they hold an earlier build's vectors, or what
the allocation held."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import BatchEngine, Engine, params, workloads
from gpumatfun_gb300.engine import GmError

pytestmark = pytest.mark.gpu

F = params.frac_exp(1e-2, 1.5)


def problem(n, R, degree):
    """diag(1 + i / n): f(A) e_i = f(1 + i / n) e_i, from one Lanczos vector."""
    return workloads.make_problem("diag", sp.diags(1.0 + np.arange(n) / n, format="csr"), np.ones((n, R)),
                                  np.zeros((n, 0)), np.zeros(0), [F] * R, 12, 32, 0.9, 2.1, degree=degree, prob_dim=0.5)


def failed_then_unit_vectors(e, n, R, rows):
    """One build with a NaN in column 0 (which leaves NaN in all its stored
    vectors, since the other columns run on), then unit vectors: solve and the
    three calls."""
    bad = np.random.default_rng(1).random((n, R))
    bad[4, 0] = np.nan
    with pytest.raises(GmError) as err:
        e.set_U(bad)
        e.solve()
    assert err.value.code == 7
    U = np.zeros((n, R))
    U[rows, np.arange(R)] = 1.0
    e.set_U(U)
    e.solve()
    meff, x = e.meff(), e.get_solution()
    e.set_U(U)
    e.build_subspace()
    e.lin_sys_solves()
    e.apply_V()
    step = e.get_solution()
    e.delete()
    np.testing.assert_array_equal(step, x)
    return U, meff, x


# the resident phase and the general one; with a polynomial and without
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
@pytest.mark.parametrize("n,R,degree,threads", [(20, 2, 0, 0), (20, 4, 2, 0), (20, 2, 0, 64), (60, 4, 3, 64)])
def test_every_column_stops_at_its_first_vector(engine_lib, precision, tol, n, R, degree, threads):
    """Against f of the eigenvalue, which the 32-node contour meets to 1e-14:
    the engine's tolerances."""
    e = Engine.from_problem(problem(n, R, degree), precision=precision, threads=threads)
    rows = [n // 2, n // 3, 7, 0][:R]
    U, meff, x = failed_then_unit_vectors(e, n, R, rows)
    assert meff == [1] * R
    assert np.abs(x - F(1.0 + np.arange(n) / n)[:, None] * U).max() < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
def test_one_problem_of_a_batch_stops(engine_lib, precision, tol):
    P = problem(40, 2, 0)
    e = BatchEngine([P, P], precision=precision, threads=64)
    bad = np.random.default_rng(1).random((80, 2))
    bad[4, 0] = np.nan
    with pytest.raises(GmError):
        e.set_U(bad)
        e.solve()
    U = np.random.default_rng(2).random((80, 2))
    U[:40] = 0.0
    U[9, 0] = U[30, 1] = 1.0
    e.set_U(U)
    e.solve()
    meff, x = e.meff(), e.get_solution()
    e.delete()
    assert meff == [1, 1, 12, 12]
    lam = 1.0 + (np.arange(80) % 40) / 40
    # the second problem's 12 vectors span its right-hand side far below 1e-6 (Chebyshev: (1/5.8)^24)
    assert np.abs(x - F(lam)[:, None] * U).max() < max(tol, 1e-9)
