"""The widest ranges of the branch-free quotients (csrc/divrn.cuh). On the GPU:
rh3t_div_check on other operands than test_gpu_math.py's. On the CPU: the tie rule of
subnormal sixths in exact arithmetic, and that the bounds which a face's and a WENO5's
range tests set give each quotient what div_near asks of it."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("exact", [True, False])
def test_bitwise(rh, exact):
    counts, first = np.zeros(7, np.int64), np.zeros(3)
    assert rh.load(exact).rh3t_div_check(0, 1_000_000_000, 11 if exact else 12, counts.ctypes.data, first.ctypes.data) == 0
    assert counts.sum() == 0, (counts.tolist(), first.tolist())


def _sixth(a, parity=True):
    """csrc/divrn.cuh div6_near in exact arithmetic on units of 2^-1074 (|a| < 2^53 units):
    q = RN(a y), then RN(q - r y'), r = 6 q - a"""
    from fractions import Fraction as F
    y = F(0x15555555555555, 2 ** 55)

    def rn(x):
        k = x.numerator // x.denominator
        f = x - k
        return k + (1 if f > F(1, 2) or (f == F(1, 2) and k % 2) else 0)

    q = rn(a * y)
    up = y + F(1, 2 ** 55) if parity and q % 2 else y
    return rn(q - (6 * q - a) * up), rn(F(a, 6))


def test_subnormal_sixths_cpu():
    """every a up to 4000 units, and large ones: the tie rule is needed and right"""
    rng = np.random.default_rng(5)
    some = list(range(4001)) + [int(x) for x in rng.integers(0, 2 ** 53, 4000)] + \
        [6 * int(k) + 3 for k in rng.integers(0, 2 ** 50, 4000)]
    wrong = 0
    for a in some:
        got, want = _sixth(a)
        assert got == want, a
        wrong += _sixth(a, parity=False)[0] != want
    assert wrong > 1000


def test_face_ranges_cpu():
    """near_face's, near_gammas' and near_eps' bounds (exponents): every numerator is 2^-969 or
    more and every quotient 2^-1000 or more, as div_near asks"""
    gk, gt, gk_most = -40, -40 + np.log2(3), 20
    for b_most, w2, vel in ((101, -800, -790), (451, -440, -430)):
        cs = (-100 - np.log2(12)) / 2
        over_b = [gk + gt + w2, 1 + gk + gt + vel, np.log2(6) + 2 * gk]
        over_c = [gk + w2, gk + vel, 2 * gk, gt + w2, 1 + gt + vel]
        # gt w2 +- 6 vel cs: zero, or a multiple of the smaller term's ulp (53 bits)
        over_c.append(min(gt + w2, np.log2(6) + vel + cs) - 53)
        assert min(over_b + over_c) >= -969
        assert min(over_b) - b_most >= -1000 and min(over_c) - 102 >= -1000
    assert gt - 800 >= -969 and gt - 800 - (gk_most + np.log2(6)) >= -1000  # R: gt w2 / (6 gk)
    lo, span = -960, 901  # WENO5: 0.1 / s over s in [lo, lo + span], and the weights' quotients
    for first in (lo, -450):
        least, most = np.log2(0.1) - (first + span), -first + 0.1
        assert least >= -969 and least - most >= -1000 and most <= 1000
