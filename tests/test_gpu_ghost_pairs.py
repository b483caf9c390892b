"""The ghost update takes heavy ghosts two to a warp: ghost values against the
oracle's where the count is odd or even, below and above the pairs one pass
over the GPU takes, for the Wall, Outflow and FarField kinds and several of them
in one launch (half-warps of one pair on different kinds and instances). The
arithmetic differs from the oracle's in pow alone (correctly rounded here):
1e-13, as for l() of the half-cylinder."""
import numpy as np
import pytest

from helpers import rel_linf

pytestmark = pytest.mark.gpu


def _cases(rh, O, name):
    if name.startswith("wall"):  # 763 (odd) and 536 Wall ghosts
        h = 1.0 / (57 if name == "wall odd" else 40)
        return rh.cases.init_double_mach(h=h), O.Case.double_mach(h=h)
    if name.startswith("planar"):  # Outflow on the right, FarField on the left, diffusion on
        nx, ny = (333, 13) if name == "planar 112" else (128, 8)
        ly = 4.0 * ny / nx
        p = dict(kappa_e=1e-3, kappa_i=1e-3, kappa_r=1e-3, omega_ei=1.0, omega_er=1.0, periodic_ly=ly)
        f = rh.cases.planar_shock(nx, ny, 4.0, ly, params=rh.Params(**p))
        return f, O.Case.planar_shock(nx=nx, ny=ny, lx=4.0, ly=ly, **p)
    h = {"far 1120": 0.1, "far 4512": 1.0 / 40.0}[name]
    return rh.cases.init_cylinder(h=h), O.Case.cylinder(h=h)


NAMES = ("wall odd", "wall even", "planar 112", "planar 72", "far 1120", "far 4512")


def _check(gv, rg, rhs, rr, fluid):
    assert rel_linf(gv, rg, np.ones(len(rg), bool)).max() <= 1e-13
    assert rel_linf(rhs, rr, fluid).max() <= 1e-13


@pytest.mark.parametrize("name", NAMES)
def test_ghost_values(rh, O, name):
    f, ref = _cases(rh, O, name)
    g = rh.GhostGrid.build(f)
    ref.run(3)
    f.value[:] = ref.state()
    f.time = ref.time
    s = rh.Solver(f, g)
    rhs, gv = s.l(with_ghosts=True)
    rr, rg = ref.l()
    _check(gv, rg, rhs, rr, f.fluid)
    s.close()


def test_mixed_batch(rh, O):
    """all of them in one launch: the pairs straddle instances and kinds"""
    fields, refs = zip(*[_cases(rh, O, n) for n in NAMES])
    for f, ref in zip(fields, refs):
        ref.run(2)
        f.value[:] = ref.state()
        f.time = ref.time
    b = rh.Batch(list(fields), [rh.GhostGrid.build(f) for f in fields])
    dt = 1e-5
    b.rk3_ssp(dt)
    for k, (f, ref) in enumerate(zip(fields, refs)):
        ref.rk3_ssp(dt)
        u, _ = b.download(k)
        assert rel_linf(u, ref.state(), f.fluid).max() <= 1e-13
    b.close()
