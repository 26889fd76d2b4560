"""Integer model of csrc/fix64.cuh's reciprocals and rounded product, against exact rationals,
and of csrc/fix64_math.cuh's log2, exp2, atan2, sin and cos (with the tables read from it),
against 60 digits and against correctly rounded floats.

The device functions restated step by step on Python integers: the third-order Newton
reciprocal of a 53-bit mantissa stays within the stated 2^5 units of 2^114 / M from every
FP32 start within two units in the last place, fix_recip_rn gives the correctly rounded
double 1 / x, and fix_mul_rn the correctly rounded double product with a float."""
import math
import random
import re
import struct
from decimal import Decimal, getcontext
from fractions import Fraction
from pathlib import Path

import pytest

MATH = Path(__file__).resolve().parents[1] / "sph_fem_2d_cutting_gpu_gb300" / "csrc" / "fix64_math.cuh"

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


def table(name):
    body = re.search(name + r"\[\d+\] = \{(.*?)\};", MATH.read_text(), re.S).group(1)
    return [int(x.rstrip("ul"), 0) for x in re.findall(r"0x[0-9a-f]+ull|\d+", body)]


def mul_hi(a, b):
    al, ah, bl, bh = a & 0xFFFFFFFF, a >> 32, b & 0xFFFFFFFF, b >> 32
    return ah * bh + ((ah * bl) >> 32) + ((al * bh) >> 32)


def umulhi(a, b):
    return (a * b) >> 32


def log2_frac(m, K, T):
    i = (m >> 56) & 0x7F
    S = ((((m >> 9) * K[i]) & M64) - (1 << 63)) << 7
    assert 0 <= S <= M64
    s = S >> 32
    h = 0x1C71C71C - (umulhi(s, 0x1999999A) >> 6)
    for c in (0x20000000, 0x24924925, 0x2AAAAAAB):
        h = c - (umulhi(s, h) >> 6)
    H = 0x3333333333333333 - (mul_hi(S, h << 32) >> 6)
    for c in (0x4000000000000000, 0x5555555555555555, 0x8000000000000000, M64):
        H = c - (mul_hi(S, H) >> 6)
    return T[i] + (mul_hi(mul_hi(S, H), 0xB8AA3B295C17F0BC) >> 5)


def exp2_frac(F, E):
    T = E[F >> 58]
    w = mul_hi((F << 6) & M64, 0xB17217F7D1CF79AC)
    v = w >> 32
    h = 0x5B05B0 + (umulhi(v, 0xD00D0) >> 6)
    for c in (0x2222222, 0xAAAAAAB):
        h = c + (umulhi(v, h) >> 6)
    H = 0x2AAAAAAAAAAAAAAB + (mul_hi(w, h << 32) >> 6)
    H = 0x8000000000000000 + (mul_hi(w, H) >> 6)
    return T + (mul_hi(T, w + mul_hi(w, mul_hi(w, H) >> 6)) >> 6)


def test_log2_exp2():
    getcontext().prec = 60
    K, T, E = table("kLog2K"), table("kLog2T"), table("kExp2T")
    two = Decimal(2)
    rng = random.Random(11)
    for k in range(6000):
        m = (1 << 52) + k if k < 1000 else (1 << 53) - 1 - k if k < 2000 else rng.getrandbits(52) | (1 << 52)
        f = log2_frac(m << 11, K, T)
        assert f <= M64 and abs(f - (Decimal(m) / (1 << 52)).ln() / two.ln() * two ** 64) < 2
        F = k if k < 1000 else M64 - k if k < 2000 else rng.getrandbits(64)
        y = exp2_frac(F, E)
        assert (1 << 63) <= y <= M64 and abs(y - two ** (Decimal(F) / (1 << 64)) * two ** 63) < 40


def to_float(m, e):
    m, e = norm(m, e)
    return math.ldexp((m >> 40) + ((m >> 39) & 1), e + 40)


def series(d2, tail, coefficients):
    d = d2 >> 32
    h = tail[1] - umulhi(d, tail[0])
    h = tail[2] - umulhi(d, h)
    H = h
    for c in coefficients:
        H = c - mul_hi(d2, H)
    return M64 - mul_hi(d2, H)


def sincosf(x):
    b = fbits(abs(x))
    if b < 0x39000000:
        return x, 1.0
    T = ((b & 0x7FFFFF) | 0x800000) << ((b >> 23) - 87)
    khi, klo = 0xC90FDAA22168C234, 0xC4C6628B80DC1CD1
    big, neg = T > khi >> 1, T > khi
    if big:
        hi, lo = ((T - khi - 1) & M64, -klo & M64) if neg else (khi - T, klo)
        z = min(64 - (hi | 1).bit_length(), 63)
        m, e = ((hi << z) | (lo >> (64 - z)) if z else hi) & M64, -63 - z
    else:
        m, e = norm(T, -63)
    dq = m >> min(-64 - e, 63)
    d2 = mul_hi(dq, dq)
    S = series(d2, (0xCA96, 0xD73F9F, 0xB092309D),
               (0x6B99159FD5, 0x2E3BC74AAD8E, 0xD00D00D00D00D, 0x222222222222222, 0x2AAAAAAAAAAAAAAB))
    C = series(d2, (0xB41, 0xD73FA, 0xC9CBA54),
               (0x8F76C77FC, 0x49F93EDDE28, 0x1A01A01A01A02, 0x5B05B05B05B05B, 0xAAAAAAAAAAAAAAB, 0x8000000000000000))
    sd, cd = to_float(mul_hi(m, S), e), to_float(C, -64)
    return math.copysign(cd if big else sd, x), ((-sd if neg else sd) if big else cd)


def atan2f(y, x, A):
    lo, hi = sorted((abs(y), abs(x)))
    lb, hb = fbits(lo), fbits(hi)
    s = (hb >> 23) - (lb >> 23)
    assert s <= 60
    ml, mh = (lb & 0x7FFFFF) | 0x800000, (hb & 0x7FFFFF) | 0x800000
    swap = abs(y) > abs(x)
    i = int(f32(f32(lo * f32(1.0 / hi)) * f32(63.9999)))
    den = mh << s if i else mh
    N, Dn = (64 * ml - i * den, 64 * den + i * ml) if i else (ml, mh)
    assert 0 <= N <= M64
    z = 64 - Dn.bit_length()
    Y = recip_mant(((Dn << z) & M64) >> 11)
    nm, ne = norm(N, 0 if i else -s) if N else (0, -63)
    qm, qe = mul_hi(nm, Y << 1), ne + z - 62
    qm, qe = norm(qm, qe) if qm else (0, qe - 63)
    z2 = mul_hi(qm, qm) >> min(-(2 * qe + 128), 63)
    h = 0x24924925 - umulhi(z2 >> 32, 0x1C71C71C)
    H = 0x3333333333333333 - mul_hi(z2, h << 32)
    H = 0x5555555555555555 - mul_hi(z2, H)
    am = mul_hi(qm, M64 - mul_hi(z2, H))
    if i == 0 and not swap and x > 0:
        return math.copysign(to_float(am, qe), y)
    sh = -61 - qe
    r = (am >> sh if sh < 64 else 0) + (A[i] >> 2)
    if swap:
        r = 0x3243F6A8885A308D - r
    if x < 0:
        r = 0x6487ED5110B4611A - r
    return math.copysign(to_float(r, -61), y)


def test_angles():
    A = table("kAtanT")
    rng = random.Random(13)
    half_pi = f32(math.pi / 2)
    for k in range(20000):
        x = (half_pi, f32(math.pi / 4))[k] if k < 2 else f32(rng.uniform(-1, 1) * half_pi * 2.0 ** -rng.choice((0, 0, 3, 12, 20)))
        if x:
            assert sincosf(x) == (f32(math.sin(x)), f32(math.cos(x)))
        y, x = f32(rng.gauss(0, 1) * 2.0 ** rng.randint(-30, 2)), f32(rng.gauss(0, 1) * 2.0 ** rng.randint(-3, 3))
        if k % 3 == 0:
            y = f32(x * rng.choice((1, -1, 1 / 64, 0.5, 63 / 64)))
        if x and y:
            assert atan2f(y, x, A) == f32(math.atan2(y, x))
