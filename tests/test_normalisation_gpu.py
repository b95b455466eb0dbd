"""The norms of the FP64 recurrence and their reciprocals.  A right-hand side
c e_i has the norm |c| and the first Lanczos vector sign(c) e_i."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import Engine, params, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [0, 64])
def test_reciprocal_norm_is_no_less_accurate_than_a_division(engine_lib, threads):
    """beta_0 and the scaled vector, 1,200 right-hand sides on the resident and the
    general path: root mean square errors no larger than with a square root and
    a division, each correctly rounded."""
    n, R = 64, 4
    A = sp.diags([-np.ones(n - 1), 2.5 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1], format="csr")
    rng = np.random.default_rng(0)
    P = workloads.make_problem("line", A, np.ones((n, R)), np.zeros((n, 0)), np.zeros(0), [params.frac_power(-0.5)] * R,
                               2, 8, 0.4, 4.6)
    e = Engine.from_problem(P, threads=threads)
    assert bool(e.info()["resident"]) == (threads == 0)
    c, beta, v = [], [], []
    for k in range(300):
        U = np.zeros((n, R))
        U[7, :] = rng.uniform(1, 4, R) * 2.0 ** rng.integers(-30, 30, R)
        e.set_U(U)
        e.build_subspace()
        c.append(U[7])
        beta.append(e.get_aabb()[0, R:])
        v.append(e.get_basis()[:, 0, 7])
    e.delete()
    c, beta, v = map(np.concatenate, (c, beta, v))
    rms = lambda x: float(np.sqrt(np.mean(x ** 2)) * 2.0 ** 53)
    norm = np.sqrt(c * c)
    unit = c * (1.0 / norm)
    assert rms(beta / c - 1) <= rms(norm / c - 1)
    assert rms(v - 1) <= rms(unit - 1)
