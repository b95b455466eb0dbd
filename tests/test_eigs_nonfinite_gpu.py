"""Deflation pairs of an operator whose products overflow."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpumatfun_gb300 import eigs
from gpumatfun_gb300.engine import GmError

pytestmark = pytest.mark.gpu


def test_overflow_is_visible(engine_lib):
    """Entries of 1.7e308: A X overflows, so the projected matrix holds NaN.
    Every Ritz value is written, as NaN, or the call reports an error: finite
    values would be what the memory held before."""
    A = sp.csr_matrix(np.full((64, 64), 1.7e308))
    import torch
    # leave recognisable numbers in memory that the call may be given
    t = [torch.full((1 << 17,), 7.0, dtype=torch.float64, device="cuda") for _ in range(64)]
    del t
    torch.cuda.empty_cache()
    try:
        lam, _, info = eigs.deflation_pairs(A, 20, max_iter=1, raise_on_noconv=False)
    except GmError:
        return
    assert not np.any(np.isfinite(lam)), lam
