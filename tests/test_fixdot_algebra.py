"""The integer arithmetic of csrc/fixdot.cuh restated in Python integers: limbs of a double, their
products and sums, the second set of limbs and the conversion back, against exact fractions."""

import random
import struct
from fractions import Fraction as F

M28 = (1 << 28) - 1
M32 = (1 << 32) - 1


def _bits(d):
    return struct.unpack("<Q", struct.pack("<d", d))[0]


def _exponent(d):
    return (_bits(d) >> 52) & 0x7FF


def limbs(d, emax):
    b = _bits(d)
    hi, lo, e = b >> 32, b & M32, _exponent(d)
    w2 = (0x80000000 | ((hi << 11) & M32) | (lo >> 21)) if e else 0
    w1, w0 = ((lo << 11) & M32) if e else 0, 0
    s = emax - e + 12
    if s >= 64:
        w0, w1, w2, s = w2, 0, 0, s - 64
    elif s >= 32:
        w0, w1, w2, s = w1, w2, 0, s - 32
    s = min(s, 32)
    r0, r1, r2 = ((w1 << 32 | w0) >> s) & M32, ((w2 << 32 | w1) >> s) & M32, w2 >> s
    sg = -1 if hi >> 31 else 1
    return (((r2 << 32 | r1) << 8 >> 32) & M32) * sg, (((r1 << 32 | r0) << 4 >> 32) & M28) * sg, (r0 & M28) * sg


def value(x, scale):
    return (F(x[0], 1 << 28) + F(x[1], 1 << 56) + F(x[2], 1 << 84)) * F(2) ** scale


def mad(s, x, y):
    return (s[0] + x[0] * y[0], s[1] + x[0] * y[1] + x[1] * y[0], s[2] + x[0] * y[2] + x[1] * y[1] + x[2] * y[0])


def sum_limbs(s):
    d = (s[1] + (s[2] >> 28)) >> 2
    h = s[0] + (d >> 26)
    return h >> 30, (h >> 2) & M28, (h & 3) << 26 | (d & ((1 << 26) - 1))


def to_double(s, scale):
    b = s[1] + (s[2] >> 28)
    h, lo = s[0] + (b >> 28), b & M28
    neg = h < 0
    if neg:
        lo = -lo & M28
        h = ~h + (lo == 0)
    if h == 0:
        if lo == 0:
            return 0.0
        h, lo, scale = lo, 0, scale - 28
    lz = 64 - h.bit_length()
    u = ((h << lz) & ((1 << 64) - 1)) | (lo >> (28 - lz) if lz <= 28 else lo << (lz - 28))
    m = ((u >> 1) + 0x200) >> 10
    e = 1023 + 63 + 28 - lz - 84 + scale
    return struct.unpack("<d", struct.pack("<Q", ((e - 1) << 52) + m + (int(neg) << 63)))[0]


def test_limbs_hold_a_double():
    r = random.Random(1)
    for _ in range(4000):
        d = r.choice([1, -1]) * r.random() * 2.0 ** r.randint(-100, 0)
        emax = max(_exponent(d), 1022)
        x = limbs(d, emax)
        assert all(abs(c) <= M28 for c in x)
        assert abs(value(x, emax - 1022) - F(d)) < F(2) ** (emax - 1022 - 84)
        if emax - _exponent(d) <= 31:  # 84 bits hold the 53 of an entry within 2^31 of the largest
            assert value(x, emax - 1022) == F(d)
    for d in (0.0, -0.0, 5e-324, 2.0 ** -1023):
        assert limbs(d, 500) == (0, 0, 0)
    for s in (0, 20, 31, 32, 51, 52, 63, 64, 83, 84, 95, 96, 200):  # every word boundary of the shift
        d = -(1.0 + 2.0 ** -52)
        assert abs(value(limbs(d, 1023 + s), s + 1) - F(d)) < F(2) ** (s + 1 - 84)


def test_products_and_sums():
    r = random.Random(2)
    for n in (1, 3, 24):
        for _ in range(600):
            a = [r.uniform(-1, 1) * 2.0 ** -r.randint(0, 24) for _ in range(n)]
            b = [r.uniform(-1, 1) * 2.0 ** -r.randint(0, 24) for _ in range(n)]
            ea, eb = max(map(_exponent, a)), max(map(_exponent, b))
            s = (0, 0, 0)
            for x, y in zip(a, b):
                s = mad(s, limbs(x, ea), limbs(y, eb))
            assert all(abs(c) < 1 << 63 for c in s)
            scale = ea + eb - 2044
            exact = sum(F(x) * F(y) for x, y in zip(a, b))
            cut = n * F(2) ** (scale - 82)
            assert abs(F(to_double(s, scale)) - exact) <= abs(exact) * F(2) ** -53 + cut
            if n == 3:
                t = sum_limbs(s)
                assert abs(t[0]) <= 1 << 28 and 0 <= t[1] <= M28 and 0 <= t[2] <= M28
                assert abs(value(t, scale + 2) - exact) <= cut


def test_sums_do_not_overflow():
    """24 products of the largest limbs, the most that an element matrix entry adds (Hex8: 8 points x 3)."""
    big = (M28, M28, M28)
    for y in (big, tuple(-c for c in big)):
        s = (0, 0, 0)
        for _ in range(24):
            s = mad(s, big, y)
        assert all(abs(c) < 1 << 63 for c in s)
