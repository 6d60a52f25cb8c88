"""The FP64 step's quotient forms (divide_by, quotient in lattice.cuh) return the correctly
rounded quotient: each fused multiply-add evaluated exactly and rounded once."""
import random
from fractions import Fraction

import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _operands(rng, n):
    for _ in range(n):
        m = rng.choice([rng.getrandbits(53), rng.getrandbits(20), (1 << 53) - 1 - rng.getrandbits(4), (1 << 52) + rng.getrandbits(4)])
        yield rng.choice([-1.0, 1.0]) * float(max(m, 1)) * 2.0 ** rng.randint(-900, 400)


@pytest.mark.parametrize("D", [6, 36, 72, 144])
def test_by_a_constant(D):
    hi = 1.0 / D
    t = 134217729.0 * hi
    a = t - (t - hi)
    b = hi - a
    lo = ((1.0 - D * a) - D * b) / D
    assert lo == float(Fraction(1, D) - Fraction(hi))
    for x in _operands(random.Random(D), 4000):
        assert _fma(x, hi, x * lo) == x / D, x.hex()
    for k in range(1, 500):  # quotients that are exact or close to a midpoint
        for x in (float(D * k), float(k), (D * k + D // 2) * 2.0 ** -52 + D):
            assert _fma(x, hi, x * lo) == x / D, x.hex()


def test_by_a_variable():
    rng = random.Random(1)
    dens = [d * 2.0 ** rng.randint(-40, 40) for d in (1.0, 1.5, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52)]
    dens += [rng.uniform(1e-3, 1.2) for _ in range(20)]
    for b in dens:
        y = 1.0 / b
        for x in _operands(rng, 300):
            a = x if abs(x) > 2.0 ** -600 else x * 2.0 ** 300
            q = a * y
            q = _fma(_fma(-b, q, a), y, q)
            q = _fma(_fma(-b, q, a), y, q)
            assert q == a / b, (a.hex(), b.hex())
