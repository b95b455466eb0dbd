"""The complex reciprocal inside the FP64 shifted solves.  With m = 1, alpha = 0,
beta_0 = 1 and the weight w, the solution for the shift -g is y = -w / g."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(lib, g, w):
    """-w / g for each g, as gm_lin_sys_solves_noalloc gives it."""
    import torch
    g, w = np.asarray(g, dtype=complex), np.asarray(w, dtype=complex)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    shifts = dev(np.stack([-g.real, -g.imag], axis=1).reshape(-1))
    wts, aabb = dev(np.concatenate([w.real, w.imag])), dev([0.0, 0.0, 1.0, 0.0])
    y = torch.full((2, g.size), np.nan, dtype=torch.float64, device="cuda")
    fn = lib.gm_lin_sys_solves_noalloc
    fn.argtypes = [ct.c_int] * 3 + [ct.c_void_p] * 7
    fn.restype = ct.c_int
    assert fn(1, 1, g.size, aabb.data_ptr(), None, wts.data_ptr(), shifts.data_ptr(), y[0].data_ptr(), y[1].data_ptr(),
              torch.cuda.current_stream().cuda_stream) == 0
    y = y.cpu().numpy()
    return y[0] + 1j * y[1]


def wide(z):
    return np.asarray(z).astype(np.clongdouble)


@pytest.mark.parametrize("exponent", [-1023, -1022, -1000, -970, 950, 960, 1000, 1019])
def test_pivots_at_the_ends_of_the_range(engine_lib, exponent):
    """g down to subnormal numbers and up to where 1/g is one.  A few roundings
    each of 2^-53, beside them the spacing of subnormal numbers, 2^-1074: of g
    relative to g, and of 1/g."""
    base = np.array([1, 1j, 3 + 1j, 1 + 3j, -5 + 2j, 1 - 7j, 4 - 4j, -2 - 6j, 1 + 0.5j])
    g = np.ldexp(base.real, exponent) + 1j * np.ldexp(base.imag, exponent)
    weight = np.ldexp(1.0, -600 if exponent < 0 else 600)
    y = solve(engine_lib, g, np.full(g.size, -weight))
    tiny = np.ldexp(np.longdouble(1.0), -1074)
    want = weight / wide(g)
    err = np.abs(wide(y) - want)
    assert np.all(err <= (8 * 2.0 ** -53 + 4 * tiny / np.abs(wide(g))) * np.abs(want) + 4 * tiny * weight)


def test_zero_and_infinite_pivots(engine_lib):
    """A singular system gives no finite solution; an infinite pivot gives 0."""
    y = solve(engine_lib, [0.0, 1.0, np.inf, 2.0j], [-1.0, -1.0, -1.0, -1.0])
    assert not np.isfinite(y[0])
    assert y[1] == 1.0 and y[2] == 0.0 and y[3] == -0.5j


def smith(a, b):
    """1 / (a + i b) by Smith's formula, each operation rounded to FP64 (the sum
    with its product in one rounding, as a fused multiply-add)."""
    big = np.abs(a) >= np.abs(b)
    x, y = np.where(big, a, b), np.where(big, b, a)
    t = y / x
    v = 1.0 / (x.astype(np.longdouble) + y.astype(np.longdouble) * t).astype(np.float64)
    return np.where(big, v, t * v) - 1j * np.where(big, t * v, v)


@pytest.mark.parametrize("spread", [(0, 0), (-10, 0), (0, -10), (-20, 20)])
def test_error_is_no_larger_than_smiths(engine_lib, spread):
    """Root mean square of the relative error over 30,000 pivots: the solves'
    error follows it.  Smith's formula has about 0.6 of 2^-53."""
    rng = np.random.default_rng(0)
    n = 30_000
    part = lambda e: rng.uniform(-1, 1, n) * 2.0 ** (rng.integers(-20, 20, n) if spread == (-20, 20) else e)
    a, b = part(spread[0]), part(spread[1])
    y = solve(engine_lib, a + 1j * b, np.full(n, -1.0))
    g = wide(a) + 1j * wide(b)
    rms = lambda z: float(np.sqrt(np.mean(np.abs(wide(z) * g - 1) ** 2)) * 2.0 ** 53)
    assert rms(smith(a, b)) < 0.7
    assert rms(y) <= rms(smith(a, b))
