"""A stencil matrix with slices of 32 empty rows: the diagonal-slice kernels
prefetch every slice's values, so a matrix with nothing to fetch in one takes
the ordinary kernels."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import Engine, params, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,no_comp", [("fp64", 0), ("mixed", 0), ("mixed", 1)])
@pytest.mark.parametrize("empty", [(), (0,), (1000, 1001), (2812,)])
def test_empty_slices(engine_lib, precision, no_comp, empty):
    """Diagonal slices (no staged columns) unless a slice is empty; the mixed
    engine's compensated diagonal fills every row.  The solution is that of the
    explicitly staged engine bit for bit."""
    n = 90_016   # 2,813 slices
    A = sp.diags([-np.ones(n - 300), -np.ones(n - 1), 4.5 * np.ones(n), -np.ones(n - 1), -np.ones(n - 300)],
                 [-300, -1, 0, 1, 300], format="csr")
    keep = np.ones(n)
    for s in empty:
        keep[32 * s:32 * s + 32] = 0.0
    A = sp.csr_matrix(sp.diags(keep) @ A @ sp.diags(keep))
    A.eliminate_zeros()
    P = workloads.make_problem("band", A, np.random.default_rng(3).random((n, 1)) * keep[:, None], np.zeros((n, 0)),
                               np.zeros(0), [params.frac_power(-0.5)], 8, 12, 0.4, 9.0, degree=2, prob_dim=2.2)
    filled = not empty or (precision == "mixed" and not no_comp)
    out = []
    for staging in (0, 2):
        e = Engine.from_problem(P, precision=precision, l2_window=1, col_staging=staging, diag_compensation=no_comp)
        e.solve()
        assert (e.info()["col_stage_groups"] == 0) == (staging == 0 and filled)
        out.append(e.get_solution())
        e.delete()
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])
