"""Deflation pairs at the edges of the kernels' layout: half a warp per row and
eight entries at a time (rows of 1 to 25 entries, odd row counts), against a
dense eigendecomposition."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import eigs

pytestmark = pytest.mark.gpu


def operator(n, width, seed):
    """Symmetric, rows of 1 (decoupled) to 2 width + 1 entries, distinct diagonal."""
    rng = np.random.default_rng(seed)
    B = sp.diags([rng.uniform(-1, 1, n - q) for q in range(1, width + 1)], list(range(1, width + 1)), shape=(n, n),
                 format="lil")
    B[: n // 8, :] = 0
    B[:, : n // 8] = 0
    B = sp.csr_matrix(B)
    B.eliminate_zeros()
    return sp.csr_matrix(B + B.T + sp.diags(4.0 * width + 3.0 * np.arange(n) + rng.uniform(0, 1, n)))


@pytest.mark.parametrize("n,width,k", [(97, 1, 1), (130, 3, 5), (257, 4, 24), (1001, 12, 7)])
@pytest.mark.parametrize("float_float", [True, False])
def test_pairs_against_dense(engine_lib, n, width, k, float_float):
    """The iteration stops at relative residuals of 1e-8, which bound the
    relative errors of the eigenvalues; vectors are orthonormal to rounding."""
    A = operator(n, width, seed=n)
    lam, Q, info = eigs.deflation_pairs(A, k, float_float_filter=float_float)
    assert info["converged"] and info["max_rel_residual"] <= 1e-8
    want = np.linalg.eigvalsh(A.toarray())[:k]
    assert np.all(np.abs(lam - want) <= 1e-8 * np.abs(want))
    assert np.abs(Q.T @ Q - np.eye(k)).max() < 1e-12
    assert (np.linalg.norm(A @ Q - Q * lam, axis=0) / np.abs(lam)).max() < 2e-8
