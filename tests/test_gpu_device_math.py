"""The arithmetic on 64-bit mantissas (csrc/fix64.cuh, csrc/fix64_math.cuh) as compiled: its functions evaluated on the
GPU element by element (device_math.cu), against exact rationals and correctly rounded doubles,
over random arguments and over the ends of their ranges."""
import ctypes as C
import math
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import build

pytestmark = pytest.mark.gpu

OPS = ("fix_double", "fix_scale", "fix_div", "div", "fix_atan2f", "atan2", "fix_sinf", "fix_cosf", "sin", "cos")


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    so = tmp_path_factory.mktemp("device_math") / "device_math.so"
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", str(build.CSRC), "-shared", str(Path(__file__).with_name("device_math.cu")),
                    "-o", str(so)], check=True)
    lib = C.CDLL(str(so))

    def call(op, a, b=None, e=None):
        a = np.ascontiguousarray(a, np.uint64)
        b = np.zeros_like(a) if b is None else np.ascontiguousarray(b, np.uint64)
        e = np.zeros(len(a), np.int32) if e is None else np.ascontiguousarray(e, np.int32)
        out = np.empty_like(a)
        r = lib.device_math(OPS.index(op), len(a), *(v.ctypes.data_as(C.c_void_p) for v in (a, b, e, out)))
        assert r == 0, f"{op}: CUDA error {r}"
        return out

    return call


def bits(x):
    return np.asarray(x, np.float64).view(np.uint64)


def nearest(f):
    """The double nearest to a rational, infinity beyond the largest."""
    try:
        return float(f)
    except OverflowError:
        return math.inf if f > 0 else -math.inf


def random_words(rng, n):
    return rng.integers(0, 1 << 64, n, dtype=np.uint64, endpoint=False)


def test_double_of_a_mantissa(evaluate):
    """Every exponent from below the subnormals to beyond the largest double."""
    rng = np.random.default_rng(1)
    e = np.concatenate([np.arange(-1200, 1100), rng.integers(-1145, -1070, 2000), rng.integers(955, 966, 200)])
    m = random_words(rng, len(e)) | np.uint64(1 << 63)
    m[::3] >>= np.uint64(7)   # not normalised
    m[1::97] = np.uint64((1 << 64) - 1)
    m[2::97] = np.uint64(1 << 63)
    m[5::97] = 0
    got = evaluate("fix_double", m, e=e).view(np.float64)
    for g, mi, ei in zip(got.tolist(), m.tolist(), e.tolist()):
        f = Fraction(mi) * Fraction(2) ** ei
        want = nearest(f)
        # ties go away from zero, to the neighbour of equal distance
        assert g == want or abs(Fraction(g) - f) == abs(Fraction(want) - f) and g > want, (mi, ei)
        assert math.copysign(1.0, g) == 1.0


def test_scaled_double(evaluate):
    """a * x with the product at and beyond both ends of the doubles; the mantissa product is short
    by less than 3 units of 2^-64 of its leading word, so the result is within 0.51 units."""
    rng = np.random.default_rng(2)
    n = 6000
    m = random_words(rng, n) | np.uint64(1 << 63)
    x = rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-1000, 1000, n).astype(np.float64)
    target = np.concatenate([rng.integers(-1090, -1010, n // 3), rng.integers(1010, 1030, n // 3),
                             rng.integers(-1200, 1200, n - 2 * (n // 3))])
    e = (target - 64 - np.frexp(x)[1]).astype(np.int32)
    x[::50] = 0.0
    x[7::50] = -0.0
    m[3::50] = 0
    got = evaluate("fix_scale", m, bits(x), e).view(np.float64)
    for g, mi, xi, ei in zip(got.tolist(), m.tolist(), x.tolist(), e.tolist()):
        f = Fraction(mi) * Fraction(xi) * Fraction(2) ** ei * (-1 if ei & 1 else 1)
        want = nearest(f)
        if math.isinf(g) or math.isinf(want) or f == 0:
            # beyond the largest double plus half a unit: infinity, with the product's sign
            assert g == want or abs(f) > Fraction(2) ** 1024 * (1 - Fraction(1, 1 << 53)), (mi, xi, ei)
        else:
            unit = Fraction(math.ulp(want))
            assert abs(Fraction(g) - f) <= Fraction(51, 100) * unit, (mi, xi, ei)
            assert g == 0.0 or (g > 0) == (f > 0)


EDGES = [0.0, -0.0, 5e-324, 2.0 ** -1022, -(2.0 ** -1023), 1.0, -1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 3.0, 0.1,
         1.7976931348623157e308, math.inf, -math.inf, math.nan] + \
        [s * 2.0 ** e * f for s in (1, -1) for e in (-512, -511, -64, -63, 63, 64, 511, 512) for f in (1.0, 1.0 - 2.0 ** -53)]


def same(a, b):
    """Equal bits, or both NaN."""
    return (a == b) | (np.isnan(a.view(np.float64)) & np.isnan(b.view(np.float64)))


def test_division(evaluate):
    """fix_div against IEEE division, bit for bit: within the ranges of its own path, where
    mantissas are equal or neighbours, and at and beyond their ends."""
    rng = np.random.default_rng(3)
    n = 2_000_000
    a, b = (rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-k, k, n).astype(np.float64)
            for k in (530, 66))
    near = rng.random(n) < 0.2
    a[near] = np.abs(b[near]) * 2.0 ** rng.integers(-20, 20, near.sum())
    a = (bits(a).astype(np.int64) + np.where(near, rng.integers(-2, 3, n), 0)).view(np.float64)
    few = rng.random(n) < 0.2   # short mantissas: exact quotients and ones beside them
    a[few], b[few] = np.rint(a[few] / 2.0 ** 500) + 1.0, np.float64(1.0) + rng.integers(0, 1000, few.sum())
    pairs = [(x, y) for x in EDGES for y in EDGES]
    a = np.concatenate([a, [p[0] for p in pairs]])
    b = np.concatenate([b, [p[1] for p in pairs]])
    got, want = evaluate("fix_div", bits(a), bits(b)), evaluate("div", bits(a), bits(b))
    bad = np.flatnonzero(~same(got, want))
    assert len(bad) == 0, [(a[i].hex(), b[i].hex(), hex(int(got[i])), hex(int(want[i]))) for i in bad[:5]]


EDGES_F = [0.0, 1e-45, 2.0 ** -149 * 3, 1.1754942e-38, 2.0 ** -126, 2.0 ** -125, 1e-20, 1.0, 1.0000001, 0.99999994, 63 / 64,
           1 / 64, 2.0 ** 60, 2.0 ** 61, 2.0 ** 125, 1.9999999 * 2.0 ** 125, 2.0 ** 126, 1.5 * 2.0 ** 126, 2.0 ** 127,
           3.4028235e38, math.inf, math.nan]


def bits_f(x):
    return np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)


def compare_floats(got, want, what, allowed):
    """Within one float of each other, and equal but for `allowed` of them; NaN and infinities equal."""
    g, w = got.astype(np.uint32).view(np.float32), want.astype(np.uint32).view(np.float32)
    finite = np.isfinite(w)
    assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(g[np.isinf(w)], w[np.isinf(w)]), what
    steps = np.abs(got.astype(np.int64) - want.astype(np.int64))[finite]   # adjacent bit patterns: adjacent floats
    assert steps.max() <= 1 and np.count_nonzero(steps) <= allowed, (what, steps.max(), np.count_nonzero(steps))


def test_atan2(evaluate):
    """fix_atan2f against the double function rounded to float.  Both round a value known to about
    2^-52 of it or better, so they differ where the value lies that close to the middle of two
    floats, once in 2^27 values: not at all in these but by chance (1.5 % in two million), so one
    is allowed.  The edges: zeros, subnormals, ratios around the table's, infinities and NaN, and
    numbers of 2^126 and more, whose reciprocal the hardware's approximation flushes to zero."""
    rng = np.random.default_rng(5)
    n = 2_000_000
    y, x = (rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n).astype(np.float64)
            for lo, hi in ((-60, 40), (-20, 40)))
    close = rng.random(n) < 0.5
    y[close] = x[close] * rng.uniform(-2.0, 2.0, close.sum())
    y, x = y.astype(np.float32), x.astype(np.float32)
    signed = [s * v for v in EDGES_F for s in (1, -1)]
    pairs = np.array([(p, q) for p in signed for q in signed], np.float32)
    for k in range(2):
        large = rng.uniform(-3.4e38, 3.4e38, (20_000, 2)).astype(np.float32)   # mostly 2^126 and more
        pairs = np.concatenate([pairs, large])
    y, x = np.concatenate([y, pairs[:, 0]]), np.concatenate([x, pairs[:, 1]])
    compare_floats(evaluate("fix_atan2f", bits_f(x), bits_f(y)), evaluate("atan2", bits_f(x), bits_f(y)), "atan2", 1)


def test_sine_and_cosine(evaluate):
    """fix_sincosf likewise, over every magnitude up to pi/2 (the half of an arctangent)."""
    rng = np.random.default_rng(6)
    half_pi = np.float32(math.pi / 2)
    x = (rng.uniform(-1.0, 1.0, 2_000_000) * half_pi).astype(np.float32)
    x[::4] *= (2.0 ** -rng.integers(1, 40, len(x[::4]))).astype(np.float32)
    near = np.arange(-2000, 1) + int(half_pi.view(np.uint32))
    quarter = np.arange(-2000, 2000) + int(np.float32(math.pi / 4).view(np.uint32))
    x = np.concatenate([x, *(v.astype(np.uint32).view(np.float32) for v in (near, quarter)),
                        np.array([0.0, -0.0, 1e-45, 2.0 ** -126, 2.0 ** -13, 2.0 ** -13 * (1 - 2.0 ** -24), -half_pi], np.float32)])
    for f in ("sin", "cos"):
        compare_floats(evaluate(f"fix_{f}f", bits_f(x)), evaluate(f, bits_f(x)), f, 1)
    bad = np.array([1.7, -2.0, 1e30, math.inf, -math.inf, math.nan], np.float32)
    for f in ("fix_sinf", "fix_cosf"):
        assert np.isnan(evaluate(f, bits_f(bad)).astype(np.uint32).view(np.float32)).all()
