"""The cell update shares each interface's jumps between its two cells and the
time-step reduction divides without a branch per quotient: l() and dt of the
no-contraction build against the oracle's, bit for bit, where tiles end short
(odd grids, every tile shape) and for mesh widths whose divisors 60 h and h lie
outside the branch-free form's range (leading fraction bits all ones). Every
operation there is IEEE in both, so the tolerance is zero on the cells that no
ghost reaches."""
import numpy as np
import pytest

from test_gpu_flux_ranges import _interior

pytestmark = pytest.mark.gpu


def _field(rh, O, nx, ny, h, source):
    f = rh.cases.rect_field(nx, ny, nx * h, ny * h, np.array([1.0, 0.0, 0.0, 1.0, 1.0, 1.0]), rh.BCType.ZEROTH_ORDER,
                            params=rh.Params(omega_ei=0.7, omega_er=0.3) if source else None)
    kw = dict(omega_ei=0.7, omega_er=0.3) if source else {}
    ref = O.Case.rect(nx, ny, nx * h, ny * h, np.array([1.0, 0.0, 0.0, 1.0, 1.0, 1.0]), kind=rh.BCType.ZEROTH_ORDER, **kw)
    x, y = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    rho = 1.0 + 0.3 * np.sin(7 * x + 3 * y)
    u, v = np.cos(5 * x - 2 * y), 0.4 * np.sin(9 * x) * np.cos(4 * y)
    p = 1.0 + 0.5 * np.sin(4 * x * y + 1.0)
    k = rho * (u * u + v * v) / 6.0
    w = np.stack([rho, rho * u, rho * v, 0.9 * p + k, 0.7 * p + k, 0.8 * p + k], -1).reshape(-1, 6)
    f.value[f.fluid] = w[f.fluid]
    ref.set_state(f.value)
    return f, ref


WIDTHS = {"1/40": 1.0 / 40.0, "sliver": float(np.nextafter(0.03125, 0.0)), "60 h sliver": float(np.nextafter(0.5, 0.0)) / 60.0}


@pytest.mark.parametrize("width", sorted(WIDTHS))
@pytest.mark.parametrize("shape", [4, 5, 6])
@pytest.mark.parametrize("nx,ny", [(33, 65), (17, 19), (70, 31)])
def test_cells(rh, O, width, shape, nx, ny):
    f, ref = _field(rh, O, nx, ny, WIDTHS[width], source=False)
    g = rh.GhostGrid.build(f)
    b = rh.Batch([f], [g], exact=True)
    b.set_tile_shapes(3, 4, shape)
    rhs = b.l(0)
    rr, _ = ref.l()
    m = _interior(f, g)
    assert m.sum() > 50 and np.array_equal(rhs[m], rr[m]), np.abs(rhs[m] - rr[m]).max(0)
    assert b.calc_global_dt()[0] == ref.global_dt()
    b.close()


@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_global_dt_ranges(rh, O, scale):
    """densities and energies inside and outside the branch-free form's range"""
    f, ref = _field(rh, O, 33, 65, 1.0 / 40.0, source=scale == 1.0)
    f.value[f.fluid] *= scale
    ref.set_state(f.value)
    s = rh.Solver(f, rh.GhostGrid.build(f))
    assert s.calc_global_dt() == ref.global_dt()
    s.close()
