"""What a step's fluxes cost must not depend on the units of the flow, on a small
eps, or on how small the velocities of gas at rest are: 8 half-cylinders of
61 x 241 in the no-contraction build, the fluxes' device time (best of 5) against
that of the same flow in the ordinary case.

The bounds. Where the branch-free form (csrc/divrn.cuh) covers the state, the
times differ by the scatter of a timing alone: 1.25. Where it does not (a gamma within
2^-40 of 1), the general form takes about twice the branch-free one's operations a
quotient, and the rest of a face's work is the same: 2. (Both forms, one after the
other, took 2.4.)"""
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


def _in_units(v, s):
    o = np.array(v, dtype=float)
    o[..., 1:3] *= s
    o[..., 3:] *= s * s
    return o


def _rest(flow, a):
    """uniform gas with velocities of size a, which stay that small"""
    f = flow[0]
    x, y = np.meshgrid(np.linspace(0, 1, f.grid.nx), np.linspace(0, 1, f.grid.ny), indexing="ij")
    e = 2.5 / 3.0 + 0.0 * x
    w = np.stack([1.0 + 0.0 * x, a * (1.0 + 0.4 * np.cos(5 * x - 2 * y)), a * np.sin(9 * x) * np.cos(4 * y), e, e, e], -1)
    w = w.reshape(-1, 6)
    w[~f.fluid] = 0.0
    return w


@pytest.mark.parametrize("case", ["2^15", "2^17", "2^20", "2^24", "2^40", "eps 1e-31", "eps 1e-40", "eps 1e-60", "eps 1e-100"])
def test_units_and_eps(rh, flow, case):
    far = rh.cases.freestream(3.0)
    ref = _flux_ms(rh, flow, flow[0].value, far, weno_q=2.0)
    if case.startswith("eps"):
        ms = _flux_ms(rh, flow, flow[0].value, far, weno_q=2.0, eps=float(case[4:]))
    else:
        s = 2.0 ** int(case[2:])
        ms = _flux_ms(rh, flow, _in_units(flow[0].value, s), _in_units(far, s), weno_q=2.0)
    assert ms <= 1.25 * ref, (ms, ref)


def test_general_form(rh, flow):
    far = rh.cases.freestream(3.0)
    ref = _flux_ms(rh, flow, flow[0].value, far, weno_q=2.0)
    ms = _flux_ms(rh, flow, flow[0].value, far, weno_q=2.0, gamma_r=1.0 + 2.0 ** -41)
    assert ms <= 2.0 * ref, (ms, ref)


@pytest.mark.parametrize("e", [-420, -1010, -1040])
def test_gas_at_rest(rh, flow, e):
    far = np.array([1.0, 0.0, 0.0, 2.5 / 3, 2.5 / 3, 2.5 / 3])
    ref = _flux_ms(rh, flow, _rest(flow, 2.0 ** -300), far)
    ms = _flux_ms(rh, flow, _rest(flow, 2.0 ** e), far)
    # velocities whose entries of L, states and averages take IEEE quotients of their own
    assert ms <= 2.2 * ref, (ms, ref)
