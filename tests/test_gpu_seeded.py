"""The FP64 reciprocal, quotients, roots, widening and comparison that the FP64
kernels use in place of CUDA's operators, against those operators and the stated
bounds: every binary exponent, both ends of the seeds' range (2^-100 .. 2^100),
significands at the ends of theirs, both signs, zeros, subnormals, infinities
and NaN."""
import ctypes as C
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from proteuscfd_gb300 import build as B

pytestmark = pytest.mark.gpu

SRC = Path(__file__).resolve().parent / "seeded_primitives.cu"
RECIP, QUOT, SHARED, ROOT, SQRT, RSQRT, WIDEN, EST, GREATER = range(9)


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    out = tmp_path_factory.mktemp("seeded") / "libseeded.so"
    subprocess.run([B._nvcc(), *B.NVCC_FLAGS, "-Xcompiler", "-fvisibility=default", "-shared", str(SRC), "-o",
                    str(out)], check=True)
    lib = C.CDLL(str(out))
    p = C.POINTER(C.c_double)

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = a if b is None else np.ascontiguousarray(b, np.float64)
        r, ref = np.empty_like(a), np.empty_like(a)
        assert lib.seeded_apply(op, C.c_longlong(a.size), *[v.ctypes.data_as(p) for v in (a, b, r, ref)]) == 0
        return r, ref
    return call


def values(n, lo, hi, seed):
    """n positive doubles with every exponent lo .. hi, one in eight with an
    extreme significand."""
    rng = np.random.default_rng(seed)
    frac = rng.integers(0, 1 << 52, size=n, dtype=np.int64)
    ends = np.array([0, 1, 2, (1 << 52) - 1, (1 << 52) - 2, 1 << 51, (1 << 29) - 1, 1 << 29], dtype=np.int64)
    pick = rng.integers(0, 8, size=n) == 0
    frac[pick] = rng.choice(ends, size=int(pick.sum()))
    exp = (np.arange(n) % (hi - lo + 1) + lo + 1023).astype(np.int64)
    return ((exp << 52) | frac).view(np.float64)


TINY = np.finfo(np.float64).tiny
SPECIAL = np.array([0.0, 5e-324, 1e-310, TINY, 1.7e308, np.inf, np.nan, 2.0 ** -100, np.nextafter(2.0 ** -100, 0),
                    2.0 ** 100, np.nextafter(2.0 ** 100, 0), 2.0 ** -127, 2.0 ** 128, 1.0, 3.0])
SPECIAL = np.concatenate([SPECIAL, -SPECIAL])


def same(r, ref):
    """equal bits, or NaN on both sides"""
    return (r.view(np.int64) == ref.view(np.int64)) | (np.isnan(r) & np.isnan(ref))


def ulps(op, r, x, y):
    """|r - the exact value| in units of the exact value's last place, exactly
    but for the last digits of a root's distance"""
    r, x, y = Fraction(r), Fraction(x), Fraction(y)
    if op in (ROOT, SQRT, RSQRT):
        # r - x^(+-1/2) from the residual: r (1 - v/r^2) / 2 to first order
        v = x if op != RSQRT else 1 / x
        err = abs((r * r - v) / (2 * r))
        exact = r
    else:
        exact = 1 / x if op == RECIP else x / y
        err = abs(r - exact)
    e = abs(exact)
    k = e.numerator.bit_length() - e.denominator.bit_length()
    while Fraction(2) ** k > e:
        k -= 1
    while Fraction(2) ** (k + 1) <= e:
        k += 1
    return float(err / Fraction(2) ** (k - 52))


@pytest.mark.parametrize("op,slack,share", [(RECIP, 2.0 ** -10, 2.0 ** -9), (QUOT, 2.0 ** -20, 2.0 ** -16),
                                            (SHARED, 2.0 ** -20, 2.0 ** -16), (ROOT, 2.0 ** -20, 2.0 ** -16),
                                            (SQRT, 0.5, 1.0), (RSQRT, 0.5, 1.0)],
                         ids=["recip", "quot", "shared", "root", "sqrt", "rsqrt"])
def test_within_the_stated_bounds(apply, op, slack, share):
    """Within half a unit of the last place and slack of one.  Where the result
    is the operator's, which rounds correctly, that holds; the others (no larger
    a share than twice slack allows) and 4,000 of all are measured exactly."""
    n = 1 << 20
    # outside its range sqrt_inv's second value is 1 / sqrt(x), rounded twice
    lo, hi = (-100, 99) if op == RSQRT else (-103, 102)
    x, y = values(n, lo, hi, 1), values(n, lo, hi, 2)
    rng = np.random.default_rng(3)
    if op in (QUOT, SHARED):
        x, y = rng.permutation(x) * rng.choice([-1.0, 1.0], n), y * rng.choice([-1.0, 1.0], n)
    r, ref = apply(op, x, y)
    other = np.flatnonzero(~same(r, ref))
    assert len(other) <= share * n
    check = np.concatenate([other[:4000], rng.integers(0, n, 4000)])
    worst = max(ulps(op, r[i], x[i], y[i]) for i in check)
    assert worst <= 0.5 + slack, worst


@pytest.mark.parametrize("op", [RECIP, QUOT, SHARED, ROOT, SQRT, RSQRT, WIDEN])
def test_operands_outside_the_range(apply, op):
    """Zeros, subnormals, infinities, NaN and both ends of the range: the
    operators' bits, in every pair for the quotients."""
    a, b = (g.ravel() for g in np.meshgrid(SPECIAL, SPECIAL, indexing="ij"))
    r, ref = apply(op, a, b)
    # inside, the forms whose bound is not the operators' rounding may differ
    # by their own unit and the operators' (1 / sqrt rounds twice)
    seeded = (a >= 2.0 ** -100) & (a < 2.0 ** 100) if op in (RECIP, SQRT, RSQRT) else np.zeros(a.shape, bool)
    with np.errstate(invalid="ignore"):
        near = seeded & (np.abs(r - ref) <= 2.0 * np.spacing(np.abs(ref)))
    assert np.all(same(r, ref) | near)


def test_widening_is_exact(apply):
    """Every exponent of FP32 with random and extreme significands, subnormals
    among them."""
    rng = np.random.default_rng(5)
    bits = (np.arange(1 << 18, dtype=np.uint32) % 512 << 23) | rng.integers(0, 1 << 23, 1 << 18, dtype=np.uint32)
    bits[::7] &= np.uint32(0xff800001)
    with np.errstate(invalid="ignore"):
        f = bits.view(np.float32).astype(np.float64)
    r, ref = apply(WIDEN, f)
    assert np.all(same(r, ref))


def test_estimates(apply):
    """Within 2^-22 in FP32's normal range, zero below it, NaN above it and for
    infinities and NaN."""
    x = np.concatenate([values(1 << 18, -200, 200, 6), SPECIAL])
    x[1::2] *= -1.0
    r, _ = apply(EST, x)
    ax = np.abs(x)
    normal = (ax >= 2.0 ** -126) & (ax < 2.0 ** 128)
    assert np.abs(r[normal] / x[normal] - 1.0).max() <= 2.0 ** -22
    assert np.all(r[ax < 2.0 ** -126] == 0.0)
    assert np.all(np.isnan(r[~(ax < 2.0 ** 128)]))


def test_integer_comparison(apply):
    """Orders every pair of numbers as the operator does, but for the zeros
    (-0 before +0)."""
    v = SPECIAL[~np.isnan(SPECIAL)]
    a, b = (g.ravel() for g in np.meshgrid(v, v, indexing="ij"))
    r, ref = apply(GREATER, a, b)
    assert np.array_equal(r, np.where((a == 0.0) & (b == 0.0), np.signbit(b) & ~np.signbit(a), ref))
