"""The small-value and FP64 forms of the division by a grid spacing (div_small, div_fast and
fdiv_f64_steps in elanfmt_gb300/csrc), restated in exact rational arithmetic: both give the IEEE
quotient, subnormal results, ties and signs included."""
from fractions import Fraction as Q

import numpy as np
import pytest


def rn(v: Q, p: int, emin: int) -> Q:
    """v rounded to p bits (ties to even) on a grid no finer than 2^emin."""
    if v == 0:
        return Q(0)
    a = abs(v)
    e = a.numerator.bit_length() - a.denominator.bit_length()
    if Q(2) ** e > a:
        e -= 1
    q = Q(2) ** max(e - p + 1, emin)
    return (-1 if v < 0 else 1) * round(a / q) * q  # round(Fraction) goes to even


def rn32(v):
    return rn(v, 24, -149)


def rn64(v):
    return rn(v, 53, -1074)


def div_fast(x, d, r, rnd, steps=1):
    q = rnd(x * r)
    for _ in range(steps):
        q = rnd(q - rnd(q * d - x) * r)
    return q


def div_small(x, d, r):
    xs = rn32(x * 2 ** 64)
    assert xs == x * 2 ** 64
    q = div_fast(xs, d, r, rn32)
    n = q * d - xs
    y = q * 2 ** 85
    Y = Q(round(y))
    if abs(y - Y) == Q(1, 2) and n != 0:
        Y = y - Q(1, 2) * (1 if n > 0 else -1)
    assert rn32(Y * Q(2) ** -149) == Y * Q(2) ** -149
    return Y * Q(2) ** -149


@pytest.mark.parametrize("dv", [40.0, 12.5, 3.0, 0.1, 33.33, 1e-3, 5e8, 1.0])
def test_small_quotients_are_ieee_quotients(dv):
    rng = np.random.default_rng(int(dv * 1000) % 9973)
    d = Q(float(np.float32(dv)))
    r = rn32(1 / d)
    xs = [Q(int(m)) * Q(2) ** -149 for m in list(range(1, 200)) + list(rng.integers(1, 1 << 23, 200))]
    for e in range(-126, -90, 3):
        xs += [Q(float(np.float32(1 + m / 2.0 ** 23))) * Q(2) ** e for m in rng.integers(0, 1 << 23, 60)]
    # quotients at and next to halves of the subnormal grid
    for m in rng.integers(1, 1 << 22, 200):
        half = (Q(int(m)) + Q(1, 2)) * Q(2) ** -149 * d
        ulp = Q(2) ** max(half.numerator.bit_length() - half.denominator.bit_length() - 24, -149)
        xs += [rn32(half), rn32(half + ulp), rn32(half - ulp)]
    for x in xs:
        if 0 < x < Q(2) ** -90:
            assert div_small(x, d, r) == rn32(x / d), (dv, float(x))
            assert div_small(-x, d, r) == rn32(-x / d)


def f64_steps(dv: float) -> int:
    r = Q(1.0 / dv)
    return 1 if abs(r * Q(dv) - 1) <= Q(2) ** -54 else 2


def test_f64_quotients_are_ieee_quotients():
    rng = np.random.default_rng(3)
    spacings = [40.0, 10.0, 11.0, 3.0, 10.3, 1 / 3.0, 1e-3] + [float(v) for v in 1.0 + rng.random(12) * 0.2]
    assert {f64_steps(v) for v in spacings} == {1, 2}
    for dv in spacings:
        d, r = Q(dv), Q(1.0 / dv)
        for sig in np.concatenate([1.0 + rng.random(150), 2.0 - rng.random(60) * 2.0 ** -40, 1.0 + rng.random(60) * 2.0 ** -40]):
            for e in (0, -700, 700):
                x = Q(float(sig)) * Q(2) ** e
                assert div_fast(x, d, r, rn64, f64_steps(dv)) == rn64(x / d), (dv, float(sig), e)
        for k in range(1, 40):  # exact quotients
            assert div_fast(d * k, d, r, rn64, f64_steps(dv)) == k
