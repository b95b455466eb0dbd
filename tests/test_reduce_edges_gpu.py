"""Block and grid sums of the general Lanczos phase at block sizes whose warps
do not fill the groups of lanes that sum them, and with more blocks than one
round of loads."""
import numpy as np
import pytest

from gpumatfun_gb300 import Engine, params, workloads
from oracle import fab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 96, 160, 352])
@pytest.mark.parametrize("R,precision", [(1, "fp64"), (2, "fp64"), (4, "fp64"), (1, "mixed"), (2, "mixed")])
def test_sums_at_odd_block_sizes(engine_lib, threads, R, precision):
    """The engine's tolerances against the oracle: 1e-10 FP64, 1e-6 mixed.
    210 x 210 rows are 1,379 slices: up to 690 blocks of two warps."""
    N = 210
    P = workloads.fd2d_problem(N, 3, 20, 16, [params.frac_exp(1e-3, 1.5)] * R, R=R, scale=(N + 1.0) ** 2, seed=R,
                               degree=2 if R == 2 else 0)
    e = Engine.from_problem(P, precision=precision, threads=threads)
    e.solve()
    x, info = e.get_solution(), e.info()
    e.delete()
    assert info["threads"] == threads and not info["resident"]
    if threads == 64:
        assert info["grid_blocks"] > 512
    want = fab.OracleEngine(A=P.A, U0=P.U, Q=P.Q, m=P.m, gamma=P.gamma, gs_re=P.gs_re, gs_im=P.gs_im, flam=P.flam,
                            wts=P.wts, shifts=P.shifts, col_scale=np.ones(R)).solve()
    assert np.linalg.norm(x - want) < (1e-10 if precision == "fp64" else 1e-6) * np.linalg.norm(want)
