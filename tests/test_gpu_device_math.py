"""The arithmetic on 64-bit mantissas (csrc/fix64.cuh, csrc/fix64_math.cuh) as compiled: its functions evaluated on the
GPU element by element (device_math.cu), against exact rationals and correctly rounded doubles,
over random arguments and over the ends of their ranges."""
import ctypes as C
import math
import subprocess
from decimal import Decimal, localcontext
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import build

pytestmark = pytest.mark.gpu

OPS = ("fix_double", "fix_scale", "fix_div", "div", "fix_atan2f", "atan2", "fix_sinf", "fix_cosf", "sin", "cos", "fix_pow",
       "pow", "fix_log_above_1", "log", "fix_pow_or_log_pow", "fix_pow_or_log_log", "rho_inv2", "rho_vol", "rho_sound",
       "float_trunc", "float_of_normal", "cand_pack64", "cand_pack32", "cand_far", "cand_row_diff")


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

    call.lib = lib
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


def units_off(got, exact):
    """Distance in units in the last place of the exact value's double."""
    return abs(Decimal(got) - exact) / Decimal(math.ulp(float(exact)))


def test_power(evaluate):
    """fix_pow within 0.6 units in its range (x > 0, 2^-9 <= n < 2, results within 2^+-32): n log2(x),
    64 bits with five before the point, is off by under five units of 2^-59, exp2 by 40 of 2^-63, so
    the value is off by under 0.1 units before its last rounding.  Outside, the library's pow."""
    rng = np.random.default_rng(7)
    n = 4000
    x = np.exp2(rng.uniform(-300.0, 300.0, n))
    x[::4] = 1.0 + rng.choice([-1, 1], len(x[::4])) * np.exp2(-rng.uniform(1.0, 52.0, len(x[::4])))
    x[1::4] = rng.uniform(0.0, 2.0, len(x[1::4]))
    k = np.exp2(rng.uniform(-9.0, 0.99, n))
    k[:6] = [2.0 ** -9, 2.0 - 2.0 ** -52, 1.0, 0.5, 1.5, 0.34]
    got, both = evaluate("fix_pow", bits(x), bits(k)), evaluate("fix_pow_or_log_pow", bits(x), bits(k))
    assert np.array_equal(got, both)
    size = np.abs(k * np.log2(x))
    own, far = size < 31.99, size > 32.01
    assert own.sum() > n // 2 and far.sum() > n // 10
    assert np.array_equal(got[far], evaluate("pow", bits(x[far]), bits(k[far])))
    with localcontext() as c:
        c.prec = 50
        for g, xi, ki in zip(got.view(np.float64)[own].tolist(), x[own].tolist(), k[own].tolist()):
            assert units_off(g, Decimal(xi) ** Decimal(ki)) <= Decimal("0.6"), (xi, ki)
    exponents = [0.0, -0.0, 2.0 ** -9 * (1 - 2.0 ** -53), 2.0, 3.0, -0.5, 300.0, math.inf, -math.inf, math.nan]
    pairs = [(p, q) for p in EDGES for q in EDGES + exponents + [0.5, 1.9]]
    a, b = (bits([p[i] for p in pairs]) for i in (0, 1))
    got, want = evaluate("fix_pow", a, b), evaluate("pow", a, b)
    assert np.array_equal(got, evaluate("fix_pow_or_log_pow", a, b))
    g, w = got.view(np.float64), want.view(np.float64)
    assert np.array_equal(np.isnan(g), np.isnan(w))
    ok = same(got, want) | (np.isfinite(w) & (np.abs(g - w) <= 2.6 * np.spacing(np.abs(w))))   # the library's own 2 units
    assert ok.all(), [(pairs[i], g[i], w[i]) for i in np.flatnonzero(~ok)[:5]]


def test_logarithm(evaluate):
    """fix_log_above_1: log2 is off by less than 2 units of 2^-64 and a truncation of 2^-64 of its
    value; with the product by ln 2 under 2^-62 in all, beside the last rounding."""
    rng = np.random.default_rng(8)
    x = np.concatenate([np.exp2(rng.uniform(0.0, 1023.0, 1500)), 1.0 + np.exp2(-rng.uniform(0.0, 52.0, 1500)),
                        [1.0 + 2.0 ** -52, 2.0, 2.0 - 2.0 ** -52, 1.7976931348623157e308]])
    got = evaluate("fix_log_above_1", bits(x))
    assert np.array_equal(got, evaluate("fix_pow_or_log_log", bits(x), bits(np.full(len(x), 0.3))))
    with localcontext() as c:
        c.prec = 50
        for g, xi in zip(got.view(np.float64).tolist(), x.tolist()):
            exact = Decimal(xi).ln()
            slack = Decimal(2) ** -62 * (1 + exact)
            assert abs(Decimal(g) - exact) <= Decimal("0.5") * Decimal(math.ulp(float(exact))) + slack, xi
    ends = bits([math.inf, math.nan])
    for op in ("fix_log_above_1", "fix_pow_or_log_log"):
        assert same(evaluate(op, ends), evaluate("log", ends)).all()


def test_density_quotients(evaluate):
    """rho_terms: 1 / rho^2 and mass / rho within 0.51 units, the root of K / rho rounded to float
    equal to the float root of the rounded quotient; densities out of range as IEEE gives them."""
    rng = np.random.default_rng(9)
    n = 3000
    rho = np.exp2(rng.uniform(-63.0, 63.0, n))
    rho[::2] = rng.uniform(1.0, 20.0, len(rho[::2]))
    mass, bulk = np.exp2(rng.uniform(-40.0, 2.0, n)), np.exp2(rng.uniform(-30.0, 30.0, n))
    out = {f: evaluate(f, bits(rho), bits(v)).view(np.float64)
           for f, v in (("rho_inv2", mass), ("rho_vol", mass), ("rho_sound", bulk))}
    for i in range(n):
        for f, exact in (("rho_inv2", 1 / Fraction(rho[i]) ** 2), ("rho_vol", Fraction(mass[i]) / Fraction(rho[i]))):
            assert abs(Fraction(out[f][i]) - exact) <= Fraction(51, 100) * Fraction(math.ulp(float(exact))), (f, rho[i])
    want = np.sqrt((bulk / rho).astype(np.float32)).astype(np.float64)
    assert np.array_equal(out["rho_sound"], want)   # once in 2^29 the two roundings of bulk / rho would differ
    with np.errstate(all="ignore"):
        r = np.array([v for v in EDGES if abs(v) > 2.0 ** 64 or not 2.0 ** -64 < abs(v) or v < 0])
        for f, m, want in (("rho_inv2", 0.5, 1.0 / (r * r)), ("rho_vol", 0.5, 0.5 / r),
                           ("rho_sound", 2.0, np.sqrt((2.0 / r).astype(np.float32)).astype(np.float64))):
            got = evaluate(f, bits(r), bits(np.full(len(r), m)))
            assert same(got, bits(want)).all(), f


def test_conversions(evaluate):
    """float_of_normal is the conversion to float; float_trunc truncates, and bounds what it cannot hold."""
    rng = np.random.default_rng(10)
    x = np.exp2(rng.uniform(-125.9, 127.0, 100_000))
    assert np.array_equal(evaluate("float_of_normal", bits(x)), bits_f(x.astype(np.float32)))
    x *= rng.choice([-1.0, 1.0], len(x))
    t = evaluate("float_trunc", bits(x)).astype(np.uint32).view(np.float32).astype(np.float64)
    assert (np.abs(t) <= np.abs(x)).all() and (np.abs(t) >= np.abs(x) * (1 - 2.0 ** -23)).all() and (t * x > 0).all()
    ends = np.array([0.0, 5e-324, 1e-300, 2.0 ** -127, 2.0 ** 127, 1e300, math.inf, math.nan, -1e300, -1e-300])
    t = evaluate("float_trunc", bits(ends)).astype(np.uint32).view(np.float32)
    assert np.array_equal(np.abs(t), np.array([0, 0, 0, 0, *[math.inf] * 5, 0], np.float32)) and t[8] < 0


def test_sigmoid_reciprocal(evaluate):
    """recip_ge1 at every float from 1 on: the correctly rounded reciprocal below 2^126, where the
    result is normal, and within one unit beyond."""
    counts, ends = (C.c_ulonglong * 2)(), (C.c_float * 2)()
    assert evaluate.lib.device_recip(counts, ends) == 0
    assert list(counts) == [0, 0] and ends[0] == 0.0 and math.isnan(ends[1])


def words(x, y):
    return bits_f(x) | (bits_f(y) << np.uint64(32))


def halves(v):
    return (v & np.uint64(0xFFFFFFFF)).astype(np.uint32).view(np.float32), (v >> np.uint64(32)).astype(np.uint32).view(np.float32)


BLANKED, NON_FINITE, FAR = 1 << 30, 1 << 28, -(1 << 31)


@pytest.mark.parametrize("cell", [4.25e-4, 8.5e-4, 1.0, 3.7e3])
def test_candidate_entries_64(evaluate, cell):
    """cand_pack64: the offsets in the cell to 8 units of the last place, the flags and the row
    (mod 8) in the lowest bits, from which cand_row_diff has the row difference up to the widest
    stencil; a record marked non-finite, or further than 4 cells off, may not be sorted out."""
    rng = np.random.default_rng(11)
    n = 40_000
    c = np.float32(cell)
    x, y = (rng.uniform(-6.0, 6.0, n).astype(np.float32) * c for _ in range(2))
    x[:4], y[4:8] = [np.nan, np.inf, -np.inf, 4 * c], [np.nan, np.inf, -np.inf, -4 * c]
    row = rng.integers(0, 5000, n).astype(np.int32)
    flags = rng.choice([0, BLANKED, NON_FINITE], n).astype(np.int32)
    v = evaluate("cand_pack64", words(x, y), bits_f(np.full(n, c)), row | flags)
    px, py = halves(v)
    low = px.view(np.uint32) & 3
    near = (np.abs(x) <= 4 * c) & (np.abs(y) <= 4 * c)
    assert np.array_equal(low & 1 == 1, flags == BLANKED)
    assert np.array_equal(low & 2 == 2, ~near | (flags == NON_FINITE))
    ok = np.isfinite(x) & np.isfinite(y)
    for p, q in ((px, x), (py, y)):
        assert (np.abs(p[ok] - q[ok]) <= 8 * np.spacing(np.abs(q[ok]))).all()
    diff = rng.integers(-3, 4, n).astype(np.int32)
    d = evaluate("cand_row_diff", bits_f(py), e=row + diff).view(np.int64)
    assert np.array_equal(d, diff)


@pytest.mark.parametrize("cell", [4.25e-4, 8.5e-4, 1.0, 3.7e3])
def test_candidate_entries_32(evaluate, cell):
    """cand_pack32: x as it is, infinite for a blanked record and NaN for one that the entry cannot
    stand for; y in the frame that repeats every 8 rows, in which two entries of a stencil have their
    distance to 2^-19 of a cell.  cand_far: further than a quarter of a cell from the cell's box."""
    rng = np.random.default_rng(12)
    n = 40_000
    c = np.float32(cell)
    edge = bits_f(np.full(n, c))
    rows, y8 = [rng.integers(3, 5000, n).astype(np.int32)], []
    rows.append(rows[0] + rng.integers(-3, 4, n).astype(np.int32))
    ys = [rng.uniform(-0.25, 1.25, n).astype(np.float32) * c for _ in rows]
    x = rng.uniform(-0.25, 1.25, n).astype(np.float32) * c
    for row, y in zip(rows, ys):
        px, py = halves(evaluate("cand_pack32", words(x, y), edge, row))
        assert np.array_equal(px, x)
        y8.append(py)
    d = np.abs(y8[0] - y8[1])
    wrapped = np.abs(np.minimum(d, np.float32(8) * c - d))
    true = np.abs((rows[0] - rows[1]) * np.float64(c) + ys[0].astype(np.float64) - ys[1])
    close = true <= 4 * np.float64(c)
    assert np.abs(wrapped[close] - true[close]).max() <= 2.0 ** -19 * cell
    assert (~close).any() and wrapped[~close].min() >= 3.4 * cell
    for flag, expect in ((BLANKED, np.isposinf), (NON_FINITE, np.isnan), (FAR, np.isnan), (BLANKED | FAR, np.isposinf)):
        e = (rows[0].astype(np.int64) | flag).astype(np.int32)
        assert expect(halves(evaluate("cand_pack32", words(x, ys[0]), edge, e))[0]).all()
    x, y = (rng.uniform(-0.6, 1.6, n).astype(np.float32) * c for _ in range(2))
    x[:4] = [np.nan, np.inf, -np.inf, 0.5 * c]
    far = evaluate("cand_far", words(x, y), edge).astype(np.uint32)
    mid = np.float32(0.5) * c
    inside = (np.abs(x - mid) <= np.float32(0.75) * c) & (np.abs(y - mid) <= np.float32(0.75) * c)
    assert np.array_equal(far, np.where(inside, 0, 1 << 31).astype(np.uint32))
