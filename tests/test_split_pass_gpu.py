"""Horner passes by (row, right-hand side) (spmv_pass_split): taken by FP64
blocks of at most five slices per warp.  Rows of 1 to 12 entries cover every
remainder of the chunks of four, two and one."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import Engine, params, workloads
from oracle import fab

pytestmark = pytest.mark.gpu


def ragged_operator(n, seed):
    """Symmetric, diagonally dominant, row lengths 1 to about 12, the first and
    last rows alone on the diagonal."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(1, max(n - 1, 1)), rng.integers(0, 6, max(n - 2, 0)))
    j = rng.integers(1, max(n - 1, 2), i.size)
    off = sp.csr_matrix((-rng.random(i.size), (i, j)), shape=(n, n))
    off = off + off.T
    off.setdiag(0.0)
    off.eliminate_zeros()
    return (off + sp.diags(np.asarray(abs(off).sum(axis=1)).ravel() + 0.5 + rng.random(n))).tocsr()


# two warps on one block: 1 slice, 10 (the last that split) with a partial one,
# 11 (by rows), then many blocks
@pytest.mark.parametrize("n,max_blocks", [(5, 1), (32, 1), (320, 1), (301, 1), (321, 1), (1500, 3), (5000, 0)])
@pytest.mark.parametrize("R,degree", [(2, 1), (2, 3), (4, 2), (4, 3)])
def test_against_oracle(engine_lib, n, max_blocks, R, degree):
    """The FP64 engine's tolerance, 1e-10 of the oracle."""
    A = ragged_operator(n, n + 50)
    U = np.random.default_rng(R).random((n, R))
    hi = float(abs(A).sum(axis=1).max())
    P = workloads.make_problem("ragged", A, U, np.zeros((n, 0)), np.zeros(0), [params.frac_power(-0.7)] * R,
                               min(8, n), 16, 0.5, hi, degree=degree)
    for kw in ({}, {"sell_sigma": 256}, {"sync_policy": 1}):
        e = Engine.from_problem(P, precision="fp64", threads=64, max_blocks=max_blocks, **kw)
        e.solve()
        x, info = e.get_solution(), e.info()
        e.delete()
        assert not info["resident"] and (max_blocks == 0 or info["grid_blocks"] <= max_blocks)
        want = fab.OracleEngine(A=P.A, U0=P.U, Q=None, m=P.m, gamma=P.gamma, gs_re=P.gs_re, gs_im=P.gs_im,
                                flam=P.flam, wts=P.wts, shifts=P.shifts, col_scale=np.ones(R)).solve()
        assert np.linalg.norm(x - want) < 1e-10 * np.linalg.norm(want)
