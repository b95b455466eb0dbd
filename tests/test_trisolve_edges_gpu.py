"""Shifted solves at the edges of their warp layout: two lanes per system, 16
systems per warp, entries loaded two ahead, warps of mixed m_eff."""
import ctypes as ct

import numpy as np
import pytest

from oracle import fab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 5, 34])
@pytest.mark.parametrize("R,C", [(1, 1), (1, 16), (2, 15), (2, 17), (4, 33)])
def test_solves_at_warp_edges(engine_lib, m, R, C):
    """Against the oracle's banded LU, with m_eff below m (and 0) in some
    columns: rows past m_eff are zero.  A solve of a well-conditioned shifted
    system (|Im sigma| >= 0.3, |T| <= 6) loses a few digits at most: 1e-10, the
    tolerance of the FP64 comparisons."""
    import torch
    rng = np.random.default_rng(100 * m + 10 * R + C)
    aabb = np.concatenate([rng.uniform(1, 3, (m + 1, R)), rng.uniform(0.5, 1.5, (m + 1, R))], axis=1)
    sigma = rng.uniform(-1, 5, R * C) + 1j * rng.uniform(0.3, 2, R * C)
    shifts = np.repeat(np.stack([sigma.real, sigma.imag], axis=1)[:, None, :], m, axis=1).reshape(-1)
    wts = [rng.standard_normal((C, 2)) for _ in range(R)]
    meff = np.array([m, max(m - 2, 0), m, 1][:R], dtype=np.int32)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    d = [dev(aabb.T.reshape(-1)), dev(meff), dev(np.concatenate([w.T.reshape(-1) for w in wts])), dev(shifts)]
    yr = torch.full((R * C, m), np.nan, dtype=torch.float64, device="cuda")
    yi = torch.full_like(yr, np.nan)
    fn = engine_lib.gm_lin_sys_solves_noalloc
    fn.argtypes = [ct.c_int] * 3 + [ct.c_void_p] * 7
    fn.restype = ct.c_int
    assert fn(m, R, C, *[t.data_ptr() for t in d], yr.data_ptr(), yi.data_ptr(),
              torch.cuda.current_stream().cuda_stream) == 0
    y = (yr + 1j * yi).cpu().numpy()
    for r in range(R):
        me, rows = int(meff[r]), slice(r * C, (r + 1) * C)
        assert np.all(y[rows, me:] == 0)
        if me:
            sh = shifts.reshape(R * C, m, 2)[rows, :me].reshape(-1)
            ore, oim = fab.tridiag_solves(aabb[:me + 1, r:r + 1].T, aabb[:me + 1, R + r:R + r + 1].T, [wts[r]], sh, m=me)
            want = (ore + 1j * oim).T
            assert np.linalg.norm(y[rows, :me] - want) <= 1e-10 * np.linalg.norm(want)
