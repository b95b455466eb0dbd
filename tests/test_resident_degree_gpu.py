"""The resident Lanczos phase on one slice (blocks of 32 threads) at the largest
polynomial degree, whose 33 coefficients are more than the block's threads."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import Engine, params, workloads
from oracle import fab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 32])
@pytest.mark.parametrize("R,degree", [(1, 31), (1, 32), (2, 32), (4, 32)])
def test_degree_32_on_one_slice(engine_lib, n, R, degree):
    """Perturbing operator, coefficients and right-hand sides by 1e-15 moves the
    oracle's result by up to 4e-9 here, so 33 Horner steps of rounding stay
    below 2e-8; a wrong last coefficient moves it by 0.4.  FP64 1e-6; the mixed
    engine has the general path's bits."""
    A = sp.diags([-np.ones(n - 1), 2.5 + 0.5 * np.arange(n) / n, -np.ones(n - 1)], [-1, 0, 1], format="csr") \
        if n > 1 else sp.csr_matrix([[2.5]])
    P = workloads.make_problem("small", A, np.random.default_rng(n).random((n, R)), np.zeros((n, 0)), np.zeros(0),
                               [params.frac_power(-0.8)] * R, min(4, n), 24, 0.4, 40.0, degree=degree, prob_dim=10.0)
    out = {}
    for precision in ("fp64", "mixed"):
        for threads in (0, 512):
            e = Engine.from_problem(P, precision=precision, threads=threads)
            e.solve()
            out[precision, threads] = e.get_solution()
            assert bool(e.info()["resident"]) == (threads == 0)
            e.delete()
    want = fab.OracleEngine(A=P.A, U0=P.U, Q=None, m=P.m, gamma=P.gamma, gs_re=P.gs_re, gs_im=P.gs_im, flam=P.flam,
                            wts=P.wts, shifts=P.shifts, col_scale=np.ones(R)).solve()
    assert np.linalg.norm(out["fp64", 0] - want) < 1e-6 * np.linalg.norm(want)
    np.testing.assert_array_equal(out["mixed", 0], out["mixed", 512])
