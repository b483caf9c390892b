"""Ghost tables whose update depends on the order of its parts (a table handed over
from another builder may be one): the ghost update of a table that GhostGrid builds
is one launch that writes ghosts while others are formed.

  - a node that is a cheap ghost and a heavy one holds the heavy ghost's value;
  - a nearest node that is not fluid is read as it was before the update: it
    holds nothing (zeros) at the first. Its L is NaN there, so that no entry of the
    first column of a Wall's system exceeds the zero of its first row: singular."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _parts(g):
    return dict(idx=g.idx.copy(), boundary=g.boundary.copy(), side=g.side.copy(), proj=g.proj.copy(),
                pre=g.pre.copy(), nearest=g.nearest.copy(), stencil=g.stencil.copy(), s=g.s.copy(), w=g.w.copy(),
                d=g.d.copy())


@pytest.fixture(scope="module")
def wedge(rh):
    """double Mach, 536 Wall ghosts, some of them on the grid below the ramp"""
    f = rh.cases.init_double_mach(h=1.0 / 40.0)
    return f, rh.GhostGrid.build(f)


@pytest.mark.parametrize("exact", [True, False])
def test_cheap_and_heavy_on_one_node(rh, wedge, exact):
    f, g = wedge
    s = rh.Solver(f, g, exact=exact)
    rhs, gv = s.l(with_ghosts=True)
    s.close()
    heavy = np.flatnonzero(g.pre >= 0)
    p = _parts(g)
    sides = [q.kind for q in f.bc_outer]
    p["idx"] = np.concatenate([p["idx"], p["idx"][heavy]])
    p["boundary"] = np.concatenate([p["boundary"], np.zeros(len(heavy), np.int32)])
    p["side"] = np.concatenate([p["side"], np.full(len(heavy), sides.index(rh.BCType.CONSTANT), np.int32)])
    p["proj"] = np.concatenate([p["proj"], p["proj"][heavy]])
    p["pre"] = np.concatenate([p["pre"], np.full(len(heavy), -1, np.int32)])
    s = rh.Solver(f, rh.GhostGrid.from_arrays(**p), exact=exact)
    n0 = s.kernel_launches
    rhs2, gv2 = s.l(with_ghosts=True)
    assert s.kernel_launches - n0 > 0
    assert np.array_equal(gv2[:len(gv)], gv) and np.array_equal(gv2[len(gv):], gv[heavy])
    assert np.array_equal(rhs2, rhs)
    a, b = rh.Solver(f, g, exact=exact), s
    b.upload(f)
    for q in (a, b):
        q.advance(3, 0.05)
    assert np.array_equal(a.download()[0], b.download()[0])
    a.close()
    b.close()


@pytest.mark.parametrize("exact", [True, False])
def test_nearest_node_not_fluid(rh, wedge, exact):
    f, g = wedge
    nx, ny = f.grid.nx, f.grid.ny
    inside = (g.idx >= 0).all(1) & (g.idx[:, 0] < nx) & (g.idx[:, 1] < ny) & (g.pre >= 0)
    assert inside.any()
    k = int(np.flatnonzero(inside)[0])
    p = _parts(g)
    p["nearest"][:] = g.idx[k]
    s = rh.Solver(f, rh.GhostGrid.from_arrays(**p), exact=exact)
    for _ in range(3):
        with pytest.raises(rh.RH3TError) as e:
            s.l()
        assert e.value.kind == "SINGULAR_ILW"
    s.close()
