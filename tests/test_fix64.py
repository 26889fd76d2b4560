"""Integer model of csrc/fix64.cuh's reciprocals and rounded product, against exact rationals.

The device functions restated step by step on Python integers: the third-order Newton
reciprocal of a 53-bit mantissa stays within the stated 2^5 units of 2^114 / M from every
FP32 start within two units in the last place, fix_recip_rn gives the correctly rounded
double 1 / x, and fix_mul_rn the correctly rounded double product with a float."""
import random
import struct
from fractions import Fraction

import pytest

M64 = (1 << 64) - 1


def dbits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def f32(x):
    return struct.unpack("<f", struct.pack("<f", x))[0]


def fbits(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


def from_fbits(b):
    return struct.unpack("<f", struct.pack("<I", b))[0]


def s64(v):
    v &= M64
    return v - (1 << 64) if v >> 63 else v


def recip_mant(M, ulps=0):
    r = f32(1.0 / from_fbits(0x3F800000 | ((M >> 29) & 0x7FFFFF)))
    r = max(min(from_fbits(fbits(r) + ulps), f32(0.99999994)), 0.5)   # the hardware's estimate may be `ulps` off
    R = (fbits(r) & 0x7FFFFF) | 0x800000
    e = s64(-(M * R))
    t = (e >> 32) * R + (((e & 0xFFFFFFFF) * R) >> 32)
    es = e >> 39
    assert abs(es) < 1 << 16   # es * es fits 32 bits
    return (R << 38) + (t >> 6) + ((R * (es * es)) >> 36)


def norm(m, e):
    z = 64 - m.bit_length()
    return m << z, e - z


def recip_rn(x, ulps):
    b = dbits(x)
    M = (b & ((1 << 52) - 1)) | (1 << 52)
    y = (recip_mant(M, ulps) + 256) >> 9
    rem = s64(-(M * y))
    y += 1 if 2 * rem > M else -1 if 2 * rem < -M else 0
    return norm(y << 10, 960 - (b >> 52))


def mul_rn(m, e, x):
    xb = fbits(x)
    xm = ((xb << 8) | 0x80000000) & 0xFFFFFFFF
    lo = xm * (m & 0xFFFFFFFF)
    p = xm * (m >> 32) + (lo >> 32)
    assert p <= M64
    rest = lo & 0xFFFFFFFF
    e = e + (xb >> 23) - 126
    if not p >> 63:
        p = ((p << 1) | (rest >> 31)) & M64
        rest = (rest << 1) & 0xFFFFFFFF
        e -= 1
    r = (p >> 11) + (((p & 0x7FF) + 0x3FF + (1 if rest or ((p >> 11) & 1) else 0)) >> 11)
    return r << 10, e + 1


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_reciprocal_and_product(ulps):
    rng = random.Random(7 + ulps)
    edges = [1 << 52, (1 << 52) + 1, (1 << 53) - 1, (1 << 53) - 2, 3 << 51]
    for k in range(20000):
        M = edges[k] if k < len(edges) else rng.getrandbits(52) | (1 << 52)
        assert abs(recip_mant(M, ulps) - Fraction(1 << 114, M)) < 32
        x = float(M) * 2.0 ** rng.randint(-70, -30)
        m, e = recip_rn(x, ulps)
        assert Fraction(m) * Fraction(2) ** e == Fraction(1 / x)
        r = f32(rng.uniform(1, 2) * 2.0 ** rng.randint(-15, 3))
        m2, e2 = mul_rn(m, e, r)
        assert Fraction(m2) * Fraction(2) ** e2 == Fraction((1 / x) * r)
