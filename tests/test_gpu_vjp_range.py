"""Operator vjp where the sum of the WENO alphas lies next to the overflow
threshold (eps 1e-154: 1 / eps^2 = 1e308), in a uniform flow and for cotangents on
cells no ghost reaches: every beta is zero there and the weights are the optimal
ones for any eps, so the cotangents equal those at eps 1e-100 to rounding (1e-12 of
their largest entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [True, False])
def test_alphas_near_overflow(rh, exact):
    def vjp(eps):
        f = rh.cases.init_cylinder(h=0.1, params=rh.Params(eps=eps, weno_q=1.0))
        b = rh.Batch([f], [rh.GhostGrid.build(f)], exact=exact)
        rbar = np.zeros(f.value.shape)
        rbar.reshape(f.grid.nx, f.grid.ny, 6)[9:13, 20:24] = np.random.default_rng(3).standard_normal((4, 4, 6))
        ub, _ = b.l_vjp(0, rbar)
        b.close()
        return ub

    want, got = vjp(1e-100), vjp(1e-154)
    assert np.abs(want).max() > 0 and np.isfinite(got).all()
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
