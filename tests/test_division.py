"""The quotient of csrc/vxb_common.cuh (divBy): x * r corrected twice by its
remainder, r the rounded reciprocal, equals the correctly rounded x / d
(Markstein 1990).  Evaluated in exact rational arithmetic with one rounding
per operation, as the fused operations round."""

import random
from fractions import Fraction

import numpy as np
import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))   # one correct rounding


def _div_by(x, d):
    r = 1.0 / d
    q = x * r
    q = _fma(_fma(-q, d, x), r, q)
    return _fma(_fma(-q, d, x), r, q)


def _mantissas(rng, n):
    # Mantissas at the ends of the binade, with few and with many set bits.
    for k in range(n):
        kind = k % 4
        if kind == 0:
            yield 1.0 + rng.getrandbits(52) * 2.0 ** -52
        elif kind == 1:
            yield 1.0 + rng.getrandbits(8) * 2.0 ** -52
        elif kind == 2:
            yield 2.0 - (1 + rng.getrandbits(8)) * 2.0 ** -52
        else:
            yield 1.0 + sum(2.0 ** -rng.randint(1, 52) for _ in range(3)) % 1.0


@pytest.mark.parametrize("scale", [0, -7, 300, -300])
def test_quotient_is_correctly_rounded(scale):
    rng = random.Random(scale)
    xs, ds = list(_mantissas(rng, 160)), list(_mantissas(rng, 160))
    for d in ds:
        d = d * 2.0 ** -scale
        for x in rng.sample(xs, 24):
            for s in (x, -x * 2.0 ** scale):
                assert _div_by(s, d) == s / d
    assert _div_by(0.0, ds[0]) == 0.0


def _round32(x):
    """A rational rounded to FP32 (nearest, ties to even), exactly."""
    f = np.float32(float(x))
    near = [f, np.nextafter(f, np.float32(np.inf)), np.nextafter(f, np.float32(-np.inf))]
    return min(near, key=lambda c: (abs(Fraction(float(c)) - x), int(c.view(np.uint32)) & 1))


def _div_by_f(x, d):
    fx, fd = Fraction(float(x)), Fraction(float(d))
    r = Fraction(float(_round32(1 / fd)))
    q = Fraction(float(_round32(fx * r)))
    for _ in range(2):
        e = Fraction(float(_round32(fx - q * fd)))
        q = Fraction(float(_round32(q + e * r)))
    return np.float32(float(q))


@pytest.mark.parametrize("scale", [0, 20, -25])
def test_float_quotient_is_correctly_rounded(scale):
    rng = random.Random(scale)
    last = np.float32(2.0 ** -23)
    ms = [np.float32(1.0 + rng.getrandbits(23) * 2.0 ** -23) for _ in range(60)]
    ms += [np.float32(1.0) + k * last for k in range(4)] + [np.float32(2.0) - k * last for k in range(1, 5)]
    for d in ms:
        for x in rng.sample(ms, 24):
            for sx in (x, -x * np.float32(2.0 ** scale)):
                assert _div_by_f(sx, d) == _round32(Fraction(float(sx)) / Fraction(float(d)))


def test_division_by_multiplication():
    """FastDiv (csrc/vxb_kernels.cuh) restated: n * m >> (27 + L) is n // d for
    every n below 2^27, with m << 4 in 32 bits."""
    rng = np.random.default_rng(1)
    ds = np.unique(np.concatenate([np.arange(2, 300), 2 ** np.arange(1, 27), 2 ** np.arange(2, 27) + 1,
                                   2 ** np.arange(2, 27) - 1, rng.integers(2, 1 << 27, 500)]))
    for d in (int(x) for x in ds):
        L = 1
        while L < 27 and (1 << L) < d:
            L += 1
        mul = ((1 << (27 + L)) // d + 1) << 4
        assert mul < 1 << 32
        top = (1 << 27) - 1
        q = top // d
        for n in {0, 1, d - 1, d, d + 1, top, q * d - 1, q * d, *(int(x) for x in rng.integers(0, 1 << 27, 20))}:
            if 0 <= n <= top:
                assert ((n * mul) >> 32) >> (L - 1) == n // d
