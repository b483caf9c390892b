"""What a step's fluxes cost must not depend on how small the velocities of gas at rest
are: 8 half-cylinders of 61 x 241 in the no-contraction build, the fluxes' device
time (best of 5) against that of the same flow in the ordinary case."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def flow(rh):
    f = rh.cases.init_cylinder(h=1.0 / 20.0)
    g = rh.GhostGrid.build(f)
    b = rh.Batch([f], [g])
    b.advance(20, 0.05)
    f.value[:] = b.download(0)[0]
    b.close()
    return f, g


def _flux_ms(rh, flow, value, far, **params):
    base, g = flow
    f = base.empty_like()
    f.value, f.time, f.params = value, 0.0, rh.Params(**params)
    f.bc_outer = [rh.BCType.FarField(far) if q.kind == rh.BCType.FAR_FIELD else q for q in base.bc_outer]
    b = rh.Batch([f] * 8, [g] * 8, exact=True)
    ms = min(b.profile_steps(2, 0.05)["flux"][0] for _ in range(5))
    b.close()
    return ms


def _rest(flow, a):
    """uniform gas with velocities of size a, which stay that small"""
    f = flow[0]
    x, y = np.meshgrid(np.linspace(0, 1, f.grid.nx), np.linspace(0, 1, f.grid.ny), indexing="ij")
    e = 2.5 / 3.0 + 0.0 * x
    w = np.stack([1.0 + 0.0 * x, a * (1.0 + 0.4 * np.cos(5 * x - 2 * y)), a * np.sin(9 * x) * np.cos(4 * y), e, e, e], -1)
    w = w.reshape(-1, 6)
    w[~f.fluid] = 0.0
    return w


@pytest.mark.parametrize("e", [-1010, -1040])
def test_gas_at_rest(rh, flow, e):
    far = np.array([1.0, 0.0, 0.0, 2.5 / 3, 2.5 / 3, 2.5 / 3])
    ref = _flux_ms(rh, flow, _rest(flow, 2.0 ** -300), far)
    ms = _flux_ms(rh, flow, _rest(flow, 2.0 ** e), far)
    # velocities whose entries of L, states and averages take IEEE quotients of their own
    assert ms <= 2.2 * ref, (ms, ref)
