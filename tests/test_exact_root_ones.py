"""The exact MPR's reciprocal of a root whose significand is all ones (inv_root in
collision-detection_b200/csrc/cc_exact_math.cuh), where Newton's steps round
wrongly and the reciprocal is put together from the root's bits instead:
the root itself, the reciprocal and the quotients by it against IEEE rounding."""
import random
import struct
from fractions import Fraction as F

import pytest

from test_exact_root import RHO, rn, root, seeds


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def from_bits(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def reciprocal(l):
    """As in inv_root, from the upper word of l."""
    return from_bits(((0x7FDFFFFF - (bits(l) >> 32)) << 32) | 1)


@pytest.mark.parametrize("k", [-100, -37, -2, -1, 0, 1, 2, 41, 99])
def test_root_reciprocal_and_quotients(k):
    rng = random.Random(k)
    l = F(2) ** k * (1 - F(1, 2 ** 53))
    assert bits(float(l)) & (2 ** 52 - 1) == 2 ** 52 - 1
    s = F(4) ** k * (1 - F(1, 2 ** 53))  # the operand with this root: (1 - u)^2 rounds to it
    assert rn(l * l) in (s, F(4) ** k * (1 - F(2, 2 ** 53)))
    y = F(reciprocal(float(l)))
    assert y == rn(1 / l) and float(y) == 1.0 / float(l)
    for r in seeds(s):
        assert root(s, r) == l
        assert abs(r * l - 1) < 2 * RHO
        for _ in range(200):
            a = F(rng.uniform(-1.0, 1.0)) * F(2) ** (k + rng.randrange(-60, 3))
            if rng.random() < 0.2:  # next to the quotients' midpoints
                a = F(float(l * (F(rng.randrange(2 ** 53, 2 ** 54) * 2 + 1, 2 ** 54))))
            q = rn(a * r)
            q = rn(q + rn(a - l * q) * r)
            q = rn(q + rn(a - l * q) * y)
            assert q == rn(a / l)
