"""The face fluxes' branch-free quotients (3t_rh_b200/csrc/divrn.cuh) and
their fallback: l() in the no-contraction build against the oracle's, bit for
bit on the cells no ghost reaches, for flows whose transverse velocity,
density or pressure lies inside, at the edge of and beyond the range that the
branch-free form accepts, and for a uniform flow (zero numerators). Every
operation there is IEEE in both, so the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _interior(f, g):
    """fluid cells whose 9-point stencils (and the faces' 6-point ones) hold fluid nodes alone"""
    nx, ny = f.grid.nx, f.grid.ny
    fl = f.fluid.reshape(nx, ny)
    out = np.zeros((nx, ny), bool)
    out[4:-4, 4:-4] = True
    for d in range(-4, 5):
        out &= np.roll(fl, d, 0) & np.roll(fl, d, 1)
    return out.reshape(-1)


# (density scale, velocity scale, pressure scale, transverse velocity): the
# branch-free form takes u, v of 0 or 2^-790..2^101, c^2 of about 2^-100..2^100
CASES = {
    "uniform": (1.0, 1.0, 1.0, None),
    "ordinary": (1.0, 1.0, 1.0, 0.3),
    "v at the edge": (1.0, 1.0, 1.0, 2.0 ** -430),
    "v below the range": (1.0, 1.0, 1.0, 2.0 ** -470),
    "v^2 subnormal": (1.0, 1.0, 1.0, 1e-160),
    "v subnormal": (1.0, 1.0, 1.0, 1e-310),
    "hot": (1.0, 1e14, 1e28, 1e14),
    "beyond the range": (1.0, 1e15, 1e31, 1e15),
    "dense": (1e12, 1.0, 1e12, 0.3),
    "thin": (1e-60, 1.0, 1e-60, 0.3),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("shape", [(2, 4, 5), (3, 6, 5), (4, 5, 4)])
def test_operator_bits(rh, O, name, shape):
    rs, us, ps, vt = CASES[name]
    f = rh.cases.init_cylinder(h=1.0 / 10.0)
    ref = O.Case.cylinder(h=1.0 / 10.0)
    g = rh.GhostGrid.build(f)
    nx, ny = f.grid.nx, f.grid.ny
    x, y = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    if vt is None:
        rho, u, v, p = 1.0 + 0 * x, 2.0 + 0 * x, 0 * x, 1.0 + 0 * x
    else:
        rho = rs * (1.0 + 0.3 * np.sin(7 * x + 3 * y))
        u = us * (1.0 + 0.4 * np.cos(5 * x - 2 * y))
        v = vt * np.sin(9 * x) * np.cos(4 * y)
        v[np.abs(y - 0.5) < 0.1] = 0.0  # exact zeros beside the others
        p = ps * (1.0 + 0.5 * np.sin(4 * x * y + 1.0))
    k = rho * (u * u + v * v) / 6.0
    w = np.stack([rho, rho * u, rho * v, p * 0.9 + k, p * 0.7 + k, p * 0.8 + k], -1).reshape(-1, 6)
    f.value[f.fluid] = w[f.fluid]
    b = rh.Batch([f], [g], exact=True)
    b.set_tile_shapes(*shape)
    rhs = b.l(0)
    ref.set_state(f.value)
    rr, _ = ref.l()
    m = _interior(f, g)
    assert m.sum() > 500
    assert np.isfinite(rr[m]).all()
    assert np.array_equal(rhs[m], rr[m]), np.abs(rhs[m] - rr[m]).max(0)
    b.close()


@pytest.mark.parametrize("nx", [128, 784, 800, 1576, 1592])
def test_thread_groups(rh, O, nx):
    """Strips with diffusion and exchange on whose flux launches have 49, 295,
    301, 592 and 598 tiles: three, three, two, two and one thread group per tile.
    As the planar shock's run: bitwise but for pow (1e-13)."""
    from helpers import rel_linf
    lx, ly = nx / 256.0, 8 / 256.0
    p = dict(kappa_e=1e-3, kappa_i=1e-3, kappa_r=1e-3, omega_ei=1.0, omega_er=1.0, periodic_ly=ly)
    f = rh.cases.planar_shock(nx, 8, lx, ly, x_shock=0.25, params=rh.Params(**p))
    ref = O.Case.planar_shock(nx=nx, ny=8, lx=lx, ly=ly, x_shock=0.25, **p)
    s = rh.Solver(f, rh.GhostGrid.build(f))
    s.advance(3, 0.05)
    ref.run(3, 0.05)
    u, _ = s.download()
    assert rel_linf(u, ref.state(), f.fluid).max() <= 1e-13
    s.close()


TINY = {"in range": 2.0 ** -788, "below it": 2.0 ** -792, "2^-878": 2.0 ** -878, "2^-882": 2.0 ** -882,
        "2^-900": 2.0 ** -900, "2^-980": 2.0 ** -980, "subnormal": 2.0 ** -1040,
        "square below 2^-800": 2.0 ** -420}


@pytest.mark.parametrize("tiny", sorted(TINY))
@pytest.mark.parametrize("which", ["u", "v", "both"])
@pytest.mark.parametrize("h", [1.0 / 10.0, 1.0 / 20.0, 1.0 / 40.0])
def test_tiny_velocities(rh, O, h, which, tiny):
    """One velocity or both falling through the range's lower end, where the
    entries of L with that velocity in the numerator are IEEE quotients; three,
    two and one thread group per tile. Bit for bit."""
    f = rh.cases.init_cylinder(h=h)
    ref = O.Case.cylinder(h=h)
    g = rh.GhostGrid.build(f)
    nx, ny = f.grid.nx, f.grid.ny
    x, y = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    rho = 1.0 + 0.3 * np.sin(7 * x + 3 * y)
    u = (TINY[tiny] if which != "v" else 1.0) * (1.0 + 0.4 * np.cos(5 * x - 2 * y))
    v = (TINY[tiny] if which != "u" else 0.7) * np.sin(9 * x) * np.cos(4 * y)
    p = 1.0 + 0.5 * np.sin(4 * x * y + 1.0)
    k = rho * (u * u + v * v) / 6.0
    w = np.stack([rho, rho * u, rho * v, p * 0.9 + k, p * 0.7 + k, p * 0.8 + k], -1).reshape(-1, 6)
    f.value[f.fluid] = w[f.fluid]
    b = rh.Batch([f], [g], exact=True)
    rhs = b.l(0)
    ref.set_state(f.value)
    rr, _ = ref.l()
    m = _interior(f, g)
    assert m.sum() > 500 and np.isfinite(rr[m]).all()
    assert np.array_equal(rhs[m], rr[m]), np.abs(rhs[m] - rr[m]).max(0)
    b.close()
