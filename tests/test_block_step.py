"""over_h (csu_b200/csrc/cuda/kernels.cuh): the division of the DPLUR blocks' finite differences by their step 1e-6 as
RN(a zh + RN(a zl)) is correctly rounded for every double in its range. The computed value lies within 2^-105 of the
quotient, so only significands whose quotient is that near to the midpoint of two doubles could round wrongly: with
A, c the 53-bit significands of dividend and step, those with |A 2^k - M c| small for an odd 54-bit M. Each is found by
inverting c modulo 2^k and checked with exact rational arithmetic, and so are random significands."""
import math
import os
import random
import re
from fractions import Fraction as Fr

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
H = 1.0e-6


def _constants():
    src = open(os.path.join(ROOT, "csu_b200", "csrc", "cuda", "kernels.cuh")).read()
    zh, zl = re.search(r"zh = (0x[0-9a-fp.+-]+), zl = (0x[0-9a-fp.+-]+);", src).groups()
    assert "constexpr double BLOCK_H = 1.0e-6;" in src
    return float.fromhex(zh), float.fromhex(zl)


def _right(a, zh, zl):
    t = float(Fr(a) * Fr(zl))                     # int and float conversions of Fraction round correctly
    return float(Fr(a) * Fr(zh) + Fr(t)) == float(Fr(a) / Fr(H))


def test_reciprocal_is_the_nearest_double_double():
    zh, zl = _constants()
    assert zh == float(1 / Fr(H)) and zl == float(1 / Fr(H) - Fr(zh)) and zl > 0


def test_every_quotient_near_a_midpoint():
    zh, zl = _constants()
    c = int(math.frexp(H)[0] * 2 ** 53)
    assert c % 2 == 1
    seen = 0
    for k in (53, 54):                            # quotient significand from A / c >= 1, and below 1
        inv = pow(c, -1, 2 ** k)
        for d in range(-64, 65):                  # |A 2^k - M c| = |d|: farther off than 2^-105 from d = 4 on
            m = (-d * inv) % 2 ** k
            while m < 2 ** 54:
                if m >= 2 ** 53 and m % 2 and (m * c + d) % 2 ** k == 0:
                    a = (m * c + d) >> k
                    if 2 ** 52 <= a < 2 ** 53:
                        seen += 1
                        assert _right(float(a), zh, zl), a
                m += 2 ** k
    assert seen > 20


def test_random_quotients():
    zh, zl = _constants()
    rng = random.Random(7)
    for _ in range(20000):
        assert _right(float(rng.randrange(2 ** 52, 2 ** 53)) * 2.0 ** rng.randint(-200, 200), zh, zl)
