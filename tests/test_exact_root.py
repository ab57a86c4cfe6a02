"""The exact MPR's root and reciprocal (inv_root in
collision-detection_b200/csrc/cc_exact_math.cuh) against IEEE rounding, on the
operands where they could fail: both formulas are emulated in exact rational
arithmetic for every approximation r of 1 / sqrt(s) within the bound the seed
step guarantees, on every operand whose result lies close enough to the
midpoint of two doubles for the formula's error to matter. All others round
correctly by the error bound alone.
"""
import math
import random
from fractions import Fraction as F

U = F(1, 2 ** 53)
RHO = F(16, 10) * U  # |r sqrt(s) - 1|


def rn(x):
    """x (> 0 or 0 or < 0) rounded to a 53-bit significand, ties to even."""
    if x == 0:
        return x
    sign, x = (1 if x > 0 else -1), abs(x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    while F(2) ** e > x:
        e -= 1
    while F(2) ** (e + 1) <= x:
        e += 1
    q = x / F(2) ** (e - 52)
    n, r = divmod(q.numerator, q.denominator)
    r = F(r, q.denominator)
    if r > F(1, 2) or (r == F(1, 2) and n & 1):
        n += 1
    return sign * n * F(2) ** (e - 52)


def test_rn_rounds_as_ieee():
    rng = random.Random(3)
    for _ in range(200):
        a, b = rng.uniform(-9, 9), rng.uniform(0.1, 9)
        assert float(rn(F(a) / F(b))) == a / b


def square_roots_mod(a, k):
    """All x in [0, 2^k) with x^2 = a mod 2^k, for a = 1 mod 8."""
    x = 1
    for i in range(3, k):
        if (x * x - a) % (1 << (i + 1)):
            x += 1 << (i - 1)
    m = 1 << k
    return {x % m, -x % m, (x + m // 2) % m, (m // 2 - x) % m}


def hard_roots():
    """s in [1, 4) whose root lies within 84 * 2^-107 / m of a midpoint m, and the
    side it lies on: S 2^54 - M^2 = D with S the integer significand of s."""
    for k, lo, hi in ((54, 2 ** 53, math.isqrt(2 ** 107) + 1), (55, math.isqrt(2 ** 107), 2 ** 54)):
        for d in range(-89, 90):
            if d % 8 != 7:  # M is odd
                continue
            for m0 in square_roots_mod(-d % (1 << k), k):
                for m in range(m0, hi + 1, 1 << k):
                    s = F((m * m + d) >> 54, 2 ** 52)
                    if m > lo and 1 <= s < 4:
                        yield s, F(m, 2 ** 53), d


def seeds(s):
    """Every double r with |r sqrt(s) - 1| <= RHO."""
    y = F(1 / math.sqrt(float(s)))
    step = F(2) ** (math.frexp(float(y))[1] - 53)
    for k in range(-6, 7):
        r = rn(y + k * step)
        if (1 - RHO) ** 2 <= r * r * s <= (1 + RHO) ** 2:
            yield r


def root(s, r):
    l0 = rn(s * r)
    return rn(l0 + rn(s - l0 * l0) * (r / 2))


def test_root_next_to_midpoints():
    tried = 0
    for s, mid, d in hard_roots():
        want = rn(mid - F(1, 2 ** 60)) if d < 0 else rn(mid + F(1, 2 ** 60))
        for r in seeds(s):
            assert root(s, r) == want, (float(s).hex(), float(r).hex())
            tried += 1
    assert tried > 50


def test_root_of_ordinary_operands():
    rng = random.Random(5)
    for _ in range(300):
        s = F(rng.uniform(1.0, 4.0))
        for r in seeds(s):
            assert float(root(s, r)) == math.sqrt(float(s))


def prime(n):
    if n < 2:
        return False
    small = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)
    for p in small:
        if n % p == 0:
            return n == p
    d, r = n - 1, 0
    while d % 2 == 0:
        d, r = d // 2, r + 1
    for a in small:
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(r - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def factors(n, rng):
    """Prime factors by Pollard's rho method."""
    if n == 1:
        return []
    if prime(n):
        return [n]
    d = 2 if n % 2 == 0 else n
    while d == n:
        x = y = rng.randrange(2, n)
        c, d = rng.randrange(1, n), 1
        while d == 1:
            x, y = (x * x + c) % n, (y * y + c) % n
            y = (y * y + c) % n
            d = math.gcd(x - y, n)
    return factors(d, rng) + factors(n // d, rng)


def step(l, y):
    return rn(y + y * rn(1 - l * y))


def test_reciprocal_of_hard_significands():
    """One step from y lands l delta^2 below 1/l (delta: the error of y; the
    residual's rounding adds at most 2^-106), so it can round wrongly only if
    2^106 - D = L M for the significand L of l, an odd 54-bit M and a small D
    (|l r - 1| <= 2.6 * 2^-53: |D| < 9): two steps from any start that r can be,
    for all such L."""
    rng = random.Random(1)
    bad = set()
    for d in (-9, -8, -7, -6, -5, -4, -3, -2, -1, 1, 2, 3, 4, 5, 6, 7, 8, 9):
        n = 2 ** 106 - d
        divisors = {1}
        for p in factors(n, rng):
            divisors |= {q * p for q in divisors}
        for L in divisors:
            if not (2 ** 52 < L < 2 ** 53 and n // L % 2 == 1 and 2 ** 53 < n // L < 2 ** 54):
                continue
            l = F(L, 2 ** 52)
            want = rn(1 / l)
            for k in range(-4, 5):
                y = want + k * U
                if abs(l * y - 1) <= F(26, 10) * U and step(l, step(l, y)) != want:
                    bad.add(L)
    assert bad <= {2 ** 53 - 1}  # all ones: sent to the slow path


def test_reciprocal_and_quotient_of_ordinary_operands():
    rng = random.Random(9)
    for _ in range(300):
        s, a = F(rng.uniform(1.0, 4.0)), F(rng.uniform(-8.0, 8.0))
        l = F(math.sqrt(float(s)))
        for r in seeds(s):
            y = step(l, step(l, r))
            assert float(y) == 1.0 / float(l)
            q = rn(a * r)
            q = rn(q + rn(a - l * q) * r)
            q = rn(q + rn(a - l * q) * y)
            assert float(q) == float(a) / float(l)
