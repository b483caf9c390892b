"""Integer powers of the boundary WENO weights (csrc/physics.cuh cr_powi) of
either sign, where the power is finite and where it overflows: eps + beta is
negative where rounding takes the quadratic form below zero, and weno_q may be
odd. Against numpy's pow, whose results here are exact or infinite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("q", [1, 2, 3, 7, 9, 10, 11, 63, 64])
def test_signed_integer_powers(rh, exact, q):
    x = np.array([2.0, -2.0, 0.5, -0.5, 1e40, -1e40, 1e308, -1e308, 2.0 ** 600, -(2.0 ** 600), np.inf, -np.inf, 0.0, -0.0])
    out = np.zeros(3 * len(x))
    assert rh.load(exact).rh3t_math_check(0, x.ctypes.data, len(x), float(q), out.ctypes.data) == 0
    got = out.reshape(-1, 3)[:, 2]
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.power(x, float(q))
        sure = (np.abs(np.log2(np.abs(x), where=x != 0, out=np.zeros_like(x))) % 1 == 0) | ~np.isfinite(want) | (x == 0)
    assert np.array_equal(got[sure], want[sure]) and np.array_equal(np.signbit(got), np.signbit(want))
    assert not np.isnan(got).any()
