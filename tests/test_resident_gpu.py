"""The resident Lanczos phase (csrc/fab_resident.cuh): problems with at most 16
slices of 32 rows per SM and every launch-shape option at its default.  An
explicit threads = 512 selects the general path for the same problem."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import Engine, params, problems, workloads
from gpumatfun_gb300.engine import GmError
from oracle import fab

pytestmark = pytest.mark.gpu

F = params.frac_exp(1e-3, 1.5)


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


def oracle(P):
    return fab.OracleEngine(A=P.A, U0=P.U, Q=P.Q if P.k else None, m=P.m, gamma=P.gamma, gs_re=P.gs_re,
                            gs_im=P.gs_im, flam=P.flam, wts=P.wts, shifts=P.shifts, col_scale=np.ones(P.R)).solve()


def run(P, **kw):
    eng = Engine.from_problem(P, **kw)
    eng.solve()
    x, info = eng.get_solution(), eng.info()
    eng.delete()
    return x, info


# one row; a partial slice; the smallest block's four slices and one more; two
# blocks; uneven blocks
@pytest.mark.parametrize("N,R,degree,precision", [
    (1, 1, 0, "fp64"), (5, 2, 1, "fp64"), (11, 4, 2, "fp64"), (12, 1, 3, "fp64"), (13, 2, 0, "mixed"),
    (37, 4, 3, "mixed"), (64, 1, 0, "fp64"), (91, 2, 5, "fp64"), (130, 4, 0, "mixed")])
def test_against_oracle_and_general_path(engine_lib, N, R, degree, precision):
    """FP64 to 1e-10 and mixed to 1e-6 of the oracle (the engine's tolerances);
    FP64 to 1e-12 of the general path, which does the same row operations and
    sums the partials in another order; mixed has its bits."""
    m = min(24, N * N)
    if N == 1:
        P = workloads.make_problem("one", sp.csr_matrix([[2.5]]), np.ones((1, 1)), np.zeros((1, 0)), np.zeros(0), [F],
                                   1, 12, 1.0, 4.0)
    else:
        P = workloads.fd2d_problem(N, min(3, N), m, 20, [F] * R, R=R, scale=(N + 1.0) ** 2, seed=N, degree=degree)
    x, info = run(P, precision=precision)
    assert info["resident"]
    g, ginfo = run(P, precision=precision, threads=512)
    assert not ginfo["resident"] and ginfo["threads"] == 512
    if precision == "mixed":
        np.testing.assert_array_equal(x, g)
    assert rel(x, g) < 1e-12
    assert rel(x, oracle(P)) < (1e-10 if precision == "fp64" else 1e-6)


def test_size_limit_and_irregular_rows(engine_lib):
    """16 slices per SM is the limit; above it the general path runs.  A mesh's
    rows of several lengths, with degree 8 and two right-hand sides."""
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    for extra, want in ((0, True), (1, False)):
        n = 16 * 32 * nsm + extra
        A = sp.diags([-np.ones(n - 1), 2.1 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1], format="csr")
        P = workloads.make_problem("line", A, np.random.default_rng(1).random((n, 1)), np.zeros((n, 0)), np.zeros(0),
                                   [params.frac_power(-0.5)], 8, 12, 0.1, 4.1)
        x, info = run(P)
        assert info["resident"] == want
        assert rel(x, oracle(P)) < 1e-10
    mesh = problems.disk_mesh(6000, seed=1)
    kappa = np.exp(problems.gaussian_random_field(mesh.nodes[mesh.tris].mean(axis=1), seed=2))
    A, ms, _ = problems.fe_operator(mesh, kappa)
    hi = float(abs(A).sum(axis=1).max())
    P = workloads.make_problem("mesh", A, np.random.default_rng(2).random((A.shape[0], 2)), np.zeros((A.shape[0], 0)),
                               np.zeros(0), [params.frac_power(-0.8)] * 2, 30, 24, 1e-5 * hi, hi, degree=8,
                               prob_dim=hi / 4, row_weight=ms)
    want = oracle(P)
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-6)):
        x, info = run(P, precision=precision)
        assert info["resident"] and rel(x, want) < tol


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("degree", [0, 4])
def test_one_way_references(engine_lib, precision, degree):
    """Blocks that are read without reading: the exchange makes them wait."""
    n = 9000
    A = sp.csr_matrix(sp.diags([2.0 * np.ones(n), np.full(n - 700, 0.1)], [0, 700]))
    P = workloads.make_problem("oneway", A, np.random.default_rng(5).random((n, 2)), np.zeros((n, 0)), np.zeros(0),
                               [F] * 2, 6, 8, 1.0, 3.0, degree=degree)
    x, info = run(P, precision=precision)
    assert info["resident"]
    for _ in range(3):
        np.testing.assert_array_equal(run(P, precision=precision)[0], x)
    assert rel(x, run(P, precision=precision, threads=512)[0]) < 1e-12


@pytest.mark.parametrize("N,R,degree", [(30, 1, 0), (100, 2, 0), (149, 4, 2), (200, 1, 3), (270, 1, 0)])
def test_mixed_keeps_the_general_paths_bits(engine_lib, N, R, degree):
    """FP32 storage amplifies last-bit changes of alpha and beta, so the mixed
    engine's sums keep the general path's groupings and trees: bit-identical
    solutions, also where a block's balanced range has more than 16 slices."""
    P = workloads.fd2d_problem(N, 0, 30, 16, [F] * R, R=R, scale=(N + 1.0) ** 2, seed=N, degree=degree)
    x, info = run(P, precision="mixed")
    assert info["resident"]
    np.testing.assert_array_equal(x, run(P, precision="mixed", threads=512)[0])


def test_breakdown_and_zero_column(engine_lib):
    """A column that spans two decoupled rows (values 1 and 3) stops at two
    vectors, a zero one at 0, and the others run on."""
    n = 1600
    T = sp.diags([-np.ones(n - 3), 2.1 * np.ones(n - 2), -np.ones(n - 3)], [-1, 0, 1])
    A = sp.csr_matrix(sp.block_diag([sp.diags([1.0, 3.0]), T]))
    U = np.random.default_rng(3).random((n, 4))
    U[:, :2] = 0.0
    U[:2, 0] = 1.0
    none = np.zeros((n, 0)), np.zeros(0)
    P = workloads.make_problem("split", A, U, *none, [F] * 4, 20, 16, 0.09, 4.2)
    eng = Engine.from_problem(P)
    eng.solve()
    x, meff, info = eng.get_solution(), eng.meff(), eng.info()
    eng.delete()
    assert info["resident"]
    assert meff == [2, 0, 20, 20]
    assert np.all(x[:, 1] == 0) and np.all(x[2:, 0] == 0)
    P1 = workloads.make_problem("split", A, U[:, 2:], *none, [F] * 2, 20, 16, 0.09, 4.2)
    assert rel(x[:, 2:], oracle(P1)) < 1e-10


def test_wait_limit_and_recovery(engine_lib):
    """With a 100 ns limit the waits of 147 blocks run out: the launch reports
    GM_ERR_TIMEOUT, and a new handle in the same context solves normally."""
    P = workloads.fd2d_problem(256, 0, 40, 16, [F], R=1, scale=257.0 ** 2, seed=4)
    with pytest.raises(GmError) as err:
        eng = Engine.from_problem(P, timeout_s=1e-7)
        for _ in range(20):
            eng.solve()
    assert err.value.code == 5
    assert rel(run(P)[0], run(P, threads=512)[0]) < 1e-12
