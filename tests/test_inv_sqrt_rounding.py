"""The rounding argument of inv_sqrt_core (csrc/walk_fp64.cuh), on the CPU in
exact arithmetic: the inputs whose square root or reciprocal lies so near the
middle of two neighbours that the sequence's error could decide are enumerated,
and each is run through the sequence with every estimate the bound allows."""
import math
from fractions import Fraction as F

# odd and even parts of 2^106 + k, |k| < 8 (a reciprocal's product d O)
FACTORS = {
    -7: [3, 3, 3, 223, 449, 30009901652533386930372133],
    -6: [2, 67, 577, 61845503, 16966443015568478977],
    -5: [19, 29, 147240723075511219048618884109],
    -4: [2, 2, 3, 5, 17, 53, 157, 1613, 2731, 8191, 858001, 308761441],
    -3: [2327027, 34864072662073401681969743],
    -2: [2, 7, 7, 31, 71, 127, 151, 337, 29191, 106681, 122921, 152041],
    -1: [3, 107, 6361, 69431, 20394401, 28059810762433],
    1: [5, 15358129, 586477649, 1801439824104653],
    2: [2, 3, 3, 11, 43, 211, 281, 331, 5419, 86171, 664441, 1564921],
    3: [13, 6951403, 306673771, 2927433831769543],
    4: [2, 2, 257, 78919881726271091143763623681],
    5: [3, 7, 140627, 173331457829, 158494480927183],
    6: [2, 5, 3366832876777, 2409672276108650191],
    7: [2269, 3253499, 10989915846903421337641],
}


def _prime(p):
    if p < 4 or p % 2 == 0:
        return p in (2, 3)
    d, s = p - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41):
        if a % p == 0:
            continue
        x = pow(a, d, p)
        if x in (1, p - 1):
            continue
        for _ in range(s - 1):
            x = x * x % p
            if x == p - 1:
                break
        else:
            return False
    return True


def _hard_roots():
    """Every x in [1, 4) with m^2 - x = k 2^-106, |k| < 48, for a middle m of
    two doubles in [1, 2): m = O 2^-53 with O odd, so O^2 = k modulo 2^54 (x
    below 2) or 2^55."""
    out = set()
    for k in range(-47, 48):
        if k % 8 != 1:  # an odd square
            continue
        for bits, lo, hi in ((54, 1, 2), (55, 2, 4)):
            roots, b = [1, 3, 5, 7], 3
            while b < bits:
                b += 1
                roots = list({t % (1 << b) for r in roots for t in (r, r + (1 << (b - 2)), r + (1 << (b - 1)))
                              if (t * t - k) % (1 << b) == 0})
            for r in roots:
                for o in range(r, 1 << 54, 1 << bits):
                    x = (o * o - k) >> 54  # in units of 2^-52
                    if o > 1 << 53 and (o * o - k) % (1 << 54) == 0 and lo << 52 <= x < hi << 52 and int(float(x)) == x:
                        out.add(x / 2.0 ** 52)
    return out


def _hard_reciprocals():
    """Every x in [1, 4) whose rounded root s = d 2^-52 has d O = 2^106 + k,
    |k| < 8, for a middle O 2^-54 of two doubles in [1/2, 1)."""
    out = set()
    for k, primes in FACTORS.items():
        n = 2 ** 106 + k
        assert math.prod(primes) == n and all(_prime(p) for p in primes)
        divisors = {1}
        for p in primes:
            divisors |= {d * p for d in divisors}
        for d in divisors:
            o = n // d
            if not (2 ** 52 <= d < 2 ** 53 and o % 2 == 1 and 2 ** 53 < o < 2 ** 54):
                continue
            lo, hi = F(2 * d - 1, 2) ** 2 / 2 ** 104, F(2 * d + 1, 2) ** 2 / 2 ** 104
            v = float(F(d * d, 2 ** 104))
            for _ in range(4):
                v = math.nextafter(v, 0.0)
            for _ in range(9):
                if lo < F(v) < hi and 1.0 <= v < 4.0:
                    out.add(v)
                v = math.nextafter(v, 8.0)
    return out


def _estimates(x):
    """The doubles y0 of 21 significant bits with |1 - x y0^2| < 2^-19."""
    c = 1.0 / math.sqrt(x)
    near = {m / 2.0 ** e for e in (21, 22) for m in range(int(c * 2 ** e) - 8, int(c * 2 ** e) + 9) if m <= 1 << 21}
    return [y for y in near if abs(1 - F(x) * F(y) ** 2) < F(1, 1 << 19)]


def _fma(a, b, c):
    return float(F(a) * F(b) + F(c))  # rounded once


def _core(x, y0):
    r = _fma(-x, y0 * y0, 1.0)
    y = _fma(_fma(r, 0.375, 0.5), y0 * r, y0)
    g = x * y
    s = _fma(_fma(-g, g, x), 0.5 * y, g)
    return _fma(_fma(-s, y, 1.0), y, y)


def _exact(x):
    k = math.isqrt(int(F(x) * 2 ** 240))
    sticky = 0 if k * k == F(x) * 2 ** 240 else 1
    s = float(F(2 * k + sticky, 2 ** 121))  # the root, rounded
    return float(1 / F(s))


def _in_range(x):
    """inv_sqrt_in_range's exclusion: the low words 0xfffffffe and 0xffffffff."""
    return int(F(x) * 2 ** (52 if x < 2.0 else 51)) & 0xffffffff < 0xfffffffe


def test_hard_cases():
    cases = _hard_roots() | _hard_reciprocals()
    assert len(cases) > 150 and 4.0 - 2.0 ** -50 in cases and 4.0 - 2.0 ** -51 in cases
    wrong = set()
    for x in cases:
        estimates = _estimates(x)
        assert estimates
        if any(_core(x, y0) != _exact(x) for y0 in estimates):
            wrong.add(x)
            assert not _in_range(x), x.hex()
    assert wrong == {4.0 - 2.0 ** -50, 4.0 - 2.0 ** -51}
