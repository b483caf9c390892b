"""The edges of the range in which a face's rows of L and R, and its WENO5s, take the
branch-free quotients (csrc/physics.cuh near_face, near_gammas, near_eps): l() in the
no-contraction build against the oracle's, bit for bit on the cells no ghost reaches,
in flows on both sides of each edge; and the ghost values there, which differ from the
oracle's in pow alone (1e-13, as in other states)."""
import numpy as np
import pytest

from helpers import rel_linf

pytestmark = pytest.mark.gpu


def _interior(f):
    nx, ny = f.grid.nx, f.grid.ny
    fl = f.fluid.reshape(nx, ny)
    out = np.zeros((nx, ny), bool)
    out[4:-4, 4:-4] = True
    for d in range(-4, 5):
        out &= np.roll(fl, d, 0) & np.roll(fl, d, 1)
    return out.reshape(-1)


def _case(rh, O, us, vs, ps, uniform=False, **params):
    """a wavy flow of velocities us, vs and pressure ps; uniform: density and pressure even"""
    f = rh.cases.init_cylinder(h=0.1, params=rh.Params(**params))
    ref = O.Case.cylinder(h=0.1, **params)
    nx, ny = f.grid.nx, f.grid.ny
    x, y = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    a = 0.0 if uniform else 1.0
    rho = 1.0 + 0.3 * a * np.sin(7 * x + 3 * y)
    u, v = us * (1.0 + 0.4 * np.cos(5 * x - 2 * y)), vs * np.sin(9 * x) * np.cos(4 * y)
    p = ps * (1.0 + 0.5 * a * np.sin(4 * x * y + 1.0))
    k = rho * (u * u + v * v) / 6.0
    g = [params.get(n, 1.4) - 1.0 for n in ("gamma_e", "gamma_i", "gamma_r")]
    w = np.stack([rho, rho * u, rho * v, p * 0.3 / g[0] + k, p * 0.4 / g[1] + k, p * 0.3 / g[2] + k], -1).reshape(-1, 6)
    f.value[f.fluid] = w[f.fluid]
    ref.set_state(f.value)
    return f, ref


def _bits(rh, f, ref, shapes=((3, 4, 4),), ghosts=False):
    rr, rg = ref.l()
    m = _interior(f)
    assert m.sum() > 500 and np.isfinite(rr[m]).all()
    b = rh.Batch([f], [rh.GhostGrid.build(f)], exact=True)
    for s in shapes:
        b.set_tile_shapes(*s)
        rhs, gv = b.l(0, with_ghosts=True)
        assert np.array_equal(rhs[m], rr[m]), np.abs(rhs[m] - rr[m]).max(0)
        if ghosts:
            assert rel_linf(gv, rg, np.ones(len(rg), bool)).max() <= 1e-13
    b.close()


# b = gt (36 ge gi gr + gt w2^2) c^2 passes 2^101 near u = c = 1e5
@pytest.mark.parametrize("speed", [5e4, 9e4, 1e5, 2e5, 1e7, 1e12, 1.5e14, 3e14])
@pytest.mark.parametrize("v", [1.0, 0.0, 2.0 ** -428, 2.0 ** -432, 2.0 ** -788, 2.0 ** -900])
def test_large_b(rh, O, speed, v):
    f, ref = _case(rh, O, speed, v * (speed if v == 1.0 else 1.0), speed ** 2)
    _bits(rh, f, ref, shapes=((3, 4, 4), (4, 6, 5)))


# gammas of 1025: b is 2^101 or more although the gas is all but at rest
@pytest.mark.parametrize("e", [-219, -221, -300, -428, -432, -600])
def test_large_b_at_rest(rh, O, e):
    f, ref = _case(rh, O, 2.0 ** e, 2.0 ** e, 1e20, gamma_e=1025.0, gamma_i=1025.0, gamma_r=1025.0)
    _bits(rh, f, ref)


@pytest.mark.parametrize("eps", [1e-31, 1e-40, 1e-66, 1e-68, 1e-100, 1e-144, 1e-145, 1e-150, 1e30, 1e67, 1e68])
@pytest.mark.parametrize("uniform", [False, True])
def test_eps(rh, O, eps, uniform):
    f, ref = _case(rh, O, 2.0, 0.3, 1.0, uniform, eps=eps, weno_q=1.0)
    _bits(rh, f, ref)


@pytest.mark.parametrize("d", [-19, -21, -38, -39, -40, -41, 19, 20, 21])
def test_gammas(rh, O, d):
    f, ref = _case(rh, O, 2.0, 0.3, 1.0, gamma_r=1.0 + 2.0 ** d)
    _bits(rh, f, ref)


@pytest.mark.parametrize("e", [-300, -420, -600, -900, -1010, -1040, -1070])
@pytest.mark.parametrize("which", ["u", "v", "both"])
def test_uniform_gas_almost_at_rest(rh, O, e, which):
    """projections and their sixths down to the last subnormals"""
    f, ref = _case(rh, O, 1.0 if which == "v" else 2.0 ** e, 1.0 if which == "u" else 2.0 ** e, 1.0, uniform=True)
    _bits(rh, f, ref, shapes=((3, 4, 4), (2, 5, 5)))


GHOSTS = {"near": dict(us=2.0, vs=0.3, ps=1.0), "large b": dict(us=1e7, vs=1e6, ps=1e14),
          "tiny velocity": dict(us=1.0, vs=2.0 ** -900, ps=1.0), "tiny square": dict(us=2.0 ** -420, vs=2.0 ** -420, ps=1.0),
          "general": dict(us=2.0, vs=0.3, ps=1.0, gamma_r=1.0 + 2.0 ** -41), "hot": dict(us=1e15, vs=1e15, ps=1e31)}


@pytest.mark.parametrize("name", sorted(GHOSTS))
def test_ghosts(rh, O, name):
    f, ref = _case(rh, O, **GHOSTS[name])
    _bits(rh, f, ref, ghosts=True)


@pytest.mark.parametrize("name", sorted(GHOSTS))
def test_ghosts_fma(rh, O, name):
    """The contracted build forms L and R by the same three routes; contraction moves L, R
    and the weights by roundings: 1e-9 of the largest value."""
    f, ref = _case(rh, O, **GHOSTS[name])
    b = rh.Batch([f], [rh.GhostGrid.build(f)], exact=False)
    _, gv = b.l(0, with_ghosts=True)
    _, rg = ref.l()
    assert rel_linf(gv, rg, np.ones(len(rg), bool)).max() <= 1e-9
    b.close()
