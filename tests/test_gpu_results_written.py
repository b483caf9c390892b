"""The calls that return new arrays write every entry of them, fluid or not:
with the memory of a new array filled with NaN beforehand none is left, and the
states and right-hand sides are what they are in zeroed memory, bit for bit
(the adjoint adds with atomics, whose order may differ between two runs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(rh):
    f = rh.cases.init_cylinder(h=0.1, params=rh.Params(omega_ei=0.5, omega_er=2.0))
    g = rh.GhostGrid.build(f)
    s = rh.Solver(f, g)
    s.advance(2, 0.05)
    out = [s.download()[0], *s.l(with_ghosts=True)]
    s.close()
    b = rh.Batch([f, f], [g, g], exact=True)
    b.advance(2, 0.05)
    out += [b.download_values()[0], b.download(1)[0], *b.l(1, with_ghosts=True)]
    rbar = np.linspace(-1.0, 1.0, f.value.size).reshape(f.value.shape)
    out.append(b.l_vjp(1, rbar)[0])
    b.adjoint_forward(2, 0.05)
    out += b.adjoint_backward([rbar, rbar])[0]
    b.close()
    return out


def test_every_entry_written(rh, monkeypatch):
    empty = np.empty
    monkeypatch.setattr(np, "empty", lambda shape, *a, **k: np.zeros(shape, *a, **k))
    ref = _calls(rh)

    def filled(shape, *a, **k):
        x = empty(shape, *a, **k)
        x.view(np.uint8).fill(0xff)
        return x

    monkeypatch.setattr(np, "empty", filled)
    got = _calls(rh)
    assert len(got) == len(ref) == 10
    for x, y in zip(got, ref):
        assert np.isfinite(y).all() and np.isfinite(x).all()
    for x, y in zip(got[:7], ref[:7]):
        assert x.tobytes() == y.tobytes()
