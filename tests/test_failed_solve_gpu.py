"""A solve that meets a non-finite value reports it and leaves the handle's
results as they were, on the resident path as on the general one."""
import ctypes as ct

import numpy as np
import pytest

from gpumatfun_gb300 import Engine, params, workloads
from gpumatfun_gb300.engine import GmError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N,threads", [(4, 0), (40, 0), (40, 128), (4, 64)])
def test_results_stay_as_they_were(engine_lib, precision, N, threads):
    P = workloads.fd2d_problem(N, 0, 10, 16, [params.frac_exp(1e-3, 1.5)], R=1, scale=(N + 1.0) ** 2, seed=2, degree=1)
    e = Engine.from_problem(P, precision=precision, threads=threads)
    e.solve()
    before = e.get_solution()
    bad = P.U.copy()
    bad[3, 0] = np.inf
    with pytest.raises(GmError) as err:
        e.set_U(bad)
        e.solve()
    assert err.value.code == 7
    out = [np.empty(P.n), np.empty(P.n)]
    for fn, dst in zip((engine_lib.gm_get_xsol, engine_lib.gm_get_solution), out):
        assert fn(e._h, dst.ctypes.data_as(ct.POINTER(ct.c_double))) == 7
    e.delete()
    np.testing.assert_array_equal(out[0], 0.0)   # set_U clears X
    np.testing.assert_array_equal(out[1], before[:, 0])
