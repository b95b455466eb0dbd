"""The adjoint on the general path, which meshes above the resident phase's
77,824 rows take: kept entry map, assembly from kappa and matrix-powers passes.
An explicit block size selects it for a small mesh."""
import numpy as np
import pytest

from gpumatfun_gb300 import adjoint, params, problems
from oracle import adjoint as oadj
from oracle import fab

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b))


# tolerances of the engine: FP64 1e-10 of the restatement; mixed as for the 2k-node gradient
@pytest.mark.parametrize("precision,tol_b,tol_k", [("fp64", 1e-10, 1e-10), ("mixed", 1e-5, 1e-4)])
@pytest.mark.parametrize("store_basis,matrix_powers", [(True, 1), (False, 1), (True, 0)])
def test_gradient_on_the_general_path(engine_lib, precision, tol_b, tol_k, store_basis, matrix_powers):
    """Against the same formula in FP64 on the oracle's Krylov state, at a kappa
    other than the one the engine was created with.  20 nodes: the lift takes eight
    to a block, and the last block has four."""
    mesh = problems.disk_mesh(1500, seed=4)
    cent = mesh.nodes[mesh.tris].mean(axis=1)
    kappa0 = np.exp(problems.gaussian_random_field(cent, sigma=1.0, ell=0.1, seed=5))
    kappa = kappa0 * np.exp(0.2 * np.sin(np.arange(kappa0.size)))
    n = int((~mesh.boundary).sum())
    rng = np.random.default_rng(6)
    b, g = rng.random(n), rng.random(n) - 0.5
    op = adjoint.FracFEOperator(mesh, kappa0, m=30, C=20, degree=5, store_basis=store_basis, precision=precision,
                                matrix_powers=matrix_powers, threads=128)
    info = op.engine.info()
    assert not info["resident"] and info["matrix_powers"] == matrix_powers and info["grid_blocks"] > 8
    t = lambda a: torch.as_tensor(a, device="cuda")
    x = op.forward(t(kappa), t(b))
    dk, db = op.backward(t(kappa), t(b), t(g))
    gs, sigma = params.shifted_poly_coeffs(op.gamma, op.contour.xi)
    w, wm = op.contour.weights(op.f), op.contour.weights_mat(op.f)
    o = fab.OracleEngine(A=op.st.matrix(kappa), U0=np.stack([b, g], axis=1), Q=None, m=op.m, gamma=op.gamma,
                         gs_re=gs.real, gs_im=gs.imag, flam=np.zeros((0, 2)), wts=[wm, wm],
                         shifts=params.shifts_vector(sigma, op.m, 2), col_scale=np.ones(2))
    o.build_subspace()
    o.lin_sys_solves()
    o.apply_V()
    xo = o.get_xsol()
    assert rel(x.cpu().numpy(), xo[:, 0]) < tol_b
    assert rel(db.cpu().numpy(), xo[:, 1]) < tol_b
    assert rel(dk.cpu().numpy(), oadj.krylov_grad(mesh, kappa, o.V, o.Yr, o.Yi, gs, w)) < tol_k
    op.delete()
