"""Diagonal slices (stencil matrices without column indices) against the
ordinary slices of the same engine, which an explicit col_staging = 2 selects:
the entries keep their order and a missing one adds zero times a finite
number, so the solutions agree bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import BatchEngine, Engine, params, problems, workloads
from oracle import fab

pytestmark = pytest.mark.gpu

F = params.frac_exp(1e-3, 1.5)


def pair(make):
    """(solution, info) with and without diagonal slices."""
    out = []
    for kw in ({}, {"col_staging": 2}):
        e = make(**kw)
        e.solve()
        out.append((e.get_solution(), e.info()))
        e.delete()
    assert out[0][1]["grid_blocks"] == out[1][1]["grid_blocks"]
    assert not out[0][1]["resident"]
    assert out[0][1]["col_stage_groups"] == 0 and out[1][1]["col_stage_groups"] > 0
    return out[0][0], out[1][0], out[0][1], out[1][1]


# the smallest grids above the resident phase's limit, odd sides: slices that
# cross lines, the first and last rows' ordinary slices, a partial slice
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("R,degree", [(1, 0), (1, 3), (2, 0), (2, 4), (4, 0), (4, 2)])
def test_2d_bit_identical(engine_lib, precision, R, degree):
    N = 281
    P = workloads.fd2d_problem(N, 3, 16, 12, [F] * R, R=R, scale=(N + 1.0) ** 2, seed=R, degree=degree)
    x, y, _, _ = pair(lambda **kw: Engine.from_problem(P, precision=precision, **kw))
    np.testing.assert_array_equal(x, y)
    if precision == "fp64":
        want = fab.OracleEngine(A=P.A, U0=P.U, Q=P.Q, m=P.m, gamma=P.gamma, gs_re=P.gs_re, gs_im=P.gs_im, flam=P.flam,
                                wts=P.wts, shifts=P.shifts, col_scale=np.ones(R)).solve()
        assert np.linalg.norm(x - want) < 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("precision,reorth", [("fp64", 0), ("fp64", 1), ("mixed", 0), ("mixed", 2)])
def test_3d_bit_identical(engine_lib, precision, reorth):
    P = workloads.fd3d_problem(45, 12, 12, [params.frac_exp(5e-4, 1.2)])
    x, y, i, j = pair(lambda **kw: Engine.from_problem(P, precision=precision, reorth=reorth, **kw))
    assert i["sell_padded"] == j["sell_padded"]
    np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("R,precision", [(1, "mixed"), (4, "mixed"), (2, "fp64")])
def test_batch_bit_identical(engine_lib, R, precision):
    """Problems start on their own slices: the row is the slot minus a shift."""
    f = [params.frac_exp(5e-6, 1.5)] * R
    probs = [workloads.fd2d_problem(N, 0, 10, 12, f, R=R, scale=(N + 1.0) ** 2, seed=N) for N in (33, 190, 7, 207, 64)]
    x, y, _, _ = pair(lambda **kw: BatchEngine(probs, precision=precision, **kw))
    np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("irregular,uses", [(0.15, True), (0.4, False)])
def test_mixture_of_slices(engine_lib, irregular, uses):
    """A band matrix with extra couplings in a share of its rows: diagonal and
    ordinary slices side by side, and the ordinary kernels below three in four."""
    n = 90_000
    rng = np.random.default_rng(7)
    A = sp.diags([-np.ones(n - 300), -np.ones(n - 1), 4.5 * np.ones(n), -np.ones(n - 1), -np.ones(n - 300)],
                 [-300, -1, 0, 1, 300], format="csr")
    rows = np.arange(int(irregular * n))
    B = sp.coo_matrix((np.full(rows.size, 0.01), (rows, rng.permutation(rows))), shape=(n, n)).tocsr()
    P = workloads.make_problem("band", sp.csr_matrix(A + B + B.T), rng.random((n, 1)), np.zeros((n, 0)), np.zeros(0),
                               [params.frac_power(-0.5)], 12, 12, 0.4, 9.0)
    for precision in ("fp64", "mixed"):
        out = []
        for kw in ({}, {"col_staging": 2}):
            e = Engine.from_problem(P, precision=precision, l2_window=1, **kw)
            e.solve()
            out.append(e.get_solution())
            if not kw:
                assert (e.info()["col_stage_groups"] == 0) == uses
            e.delete()
        np.testing.assert_array_equal(out[0], out[1])
