"""The FP64 arithmetic that the ref and fp64 kernels do off the FP64 pipe, function by function over random
operands of the whole range, operands near the powers of two, and zeros, subnormals, infinities and NaN.

Conversions, halves, blends, minima and comparisons are those of IEEE arithmetic to the bit, signs of zero
included, and so is the division (a remainder-corrected quotient).  The reciprocal is one third-order step in
FP64 from a seed of 22 bits or more: the step leaves 2^-66, the last rounding half an ulp, so 0.5 + 2^-12 ulp.
The reciprocal root rounds x y0 once more, 2^-53 of the correction's 1/2: at most 0.5 ulp on top, 1 + 2^-10.
Operands outside the seeds' range take CUDA's own operations: the division exact, rsqrt within 1 ulp."""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

RCP, RSQRT, DIV, TO_FLOAT, TO_DOUBLE, HALF, FIRST, SECOND, MAX, MIN, TOP, COMPARE = range(12)


@pytest.fixture(scope="module")
def pairs():
    if not gpu_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(11)
    n = 400_000

    def wide():  # any bits: every exponent, NaN and infinities among them
        return rng.integers(0, 2 ** 64, n, dtype=np.uint64).view(np.float64)

    def flow():  # what a flow field holds
        return rng.choice([-1.0, 1.0], n) * np.exp(rng.uniform(-30.0, 30.0, n))

    def near():  # a few ulp from powers of two and from halves of FP32 ulps
        x = np.ldexp(1.0, rng.integers(-1074, 1024, n)).view(np.uint64)
        step = rng.choice(np.array([0, 1, 2, 3, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 1, 2 ** 29 - 1, 2 ** 29], dtype=np.uint64), n)
        x = np.where(rng.random(n) < 0.5, x + step, x - np.minimum(x, step))
        return x.view(np.float64) * rng.choice([-1.0, 1.0], n)

    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308, 1.797e308, 1.0, -1.0,
                        3.4028234663852886e38, 3.4028235677973366e38, 1.1754943508222875e-38, 1.4e-45, 0.5, 2.0])
    sa, sb = (x.ravel() for x in np.meshgrid(special, special))
    a = np.concatenate([wide(), flow(), near(), flow(), sa])
    b = np.concatenate([wide(), flow(), near(), near(), sb])
    return a, b


def device(op, a, b):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import _ffi

    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    out = np.empty_like(a)
    p = [C.c_void_p(x.ctypes.data) for x in (a, b, out)]
    _ffi.check(_ffi.lib().afar_debug_arithmetic(0, op, a.size, *p))
    return out


def same_bits(x, y):
    """Equal to the bit; any NaN is any other."""
    ok = (x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))
    bad = np.flatnonzero(~ok)
    assert bad.size == 0, [(int(i), float(x[i]).hex(), float(y[i]).hex()) for i in bad[:5]]


@pytest.mark.parametrize("op", [DIV, TO_FLOAT, TO_DOUBLE, HALF, FIRST, SECOND, MAX, MIN, COMPARE])
def test_to_the_bit(pairs, op):
    a, b = pairs
    with np.errstate(all="ignore"):
        if op == DIV:
            want = a / b
        elif op in (TO_FLOAT, TO_DOUBLE):
            want = a.astype(np.float32).astype(np.float64)
        elif op == HALF:
            want = a * 0.5
        elif op == FIRST:
            want = 1.0 * a + 0.0 * b
        elif op == SECOND:
            want = 0.0 * a + 1.0 * b
        elif op in (MAX, MIN):
            quiet = [np.where(np.isnan(x), np.nan, x) for x in (a, b)]  # (numpy's return a signalling NaN)
            want = (np.fmax if op == MAX else np.fmin)(*quiet)
            zeros = (a == 0.0) & (b == 0.0)  # either zero
            got = device(op, a, b)
            assert (got[zeros] == 0.0).all()
            same_bits(got[~zeros], want[~zeros])
            return
        else:
            b = np.abs(np.where(np.isnan(b) | (b == 0.0), 1e-5, b))  # compared with positive constants
            nan = (a.view(np.uint64) >> np.uint64(32)) & np.uint64(0x7FFFFFFF) > np.uint64(0x7FF00000)
            keep = ~np.isnan(a) | nan  # a NaN of the lower bits alone does not come out of arithmetic
            a, b, nan = a[keep], b[keep], nan[keep]
            want = (a > 0) + 2.0 * (a <= 0) + 4.0 * (np.abs(a) < b) + 8.0 * (np.abs(a) >= b) + 16.0 * nan
    same_bits(device(op, a, b), want.astype(np.float64))


@pytest.mark.parametrize("op,ulps", [(RCP, 0.5 + 2.0 ** -12), (RSQRT, 1.0 + 2.0 ** -10)])
def test_within_its_bound(pairs, op, ulps):
    a, b = pairs
    got = device(op, a, b)
    with np.errstate(all="ignore"):
        want = 1.0 / a if op == RCP else 1.0 / np.sqrt(a)
        plain = np.isfinite(want) & (np.abs(want) >= 2.2250738585072014e-308) & np.isfinite(a)
        same_bits(got[~plain & (want != 0.0) & ~np.isfinite(want)], want[~plain & (want != 0.0) & ~np.isfinite(want)])
        assert (got[want == 0.0] == 0.0).all()
        x, y = a[plain].astype(np.longdouble), got[plain]
        ref = 1 / x if op == RCP else 1 / np.sqrt(x)
        err = np.abs(y.astype(np.longdouble) - ref) / np.spacing(np.abs(ref.astype(np.float64))).astype(np.longdouble)
    # (an ulp that shrinks at the power of two below the value counts twice)
    worst = int(np.argmax(err))
    assert err[worst] <= ulps, (float(a[plain][worst]).hex(), float(err[worst]))


def test_top_float_has_twenty_bits(pairs):
    a, b = pairs
    got = device(TOP, a, b)
    mag = np.abs(a)
    inside = np.isfinite(a) & (mag >= 2.0 ** -126) & (mag < 2.0 ** 128)
    assert (np.abs(got[inside] - a[inside]) <= 2.0 ** -20 * mag[inside]).all()
    assert (got[mag < 2.0 ** -126] == 0.0).all()
    large = mag >= 2.0 ** 128
    assert (got[large] == np.copysign(np.inf, a[large])).all()


def test_unknown_operations_are_refused():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import _ffi

    x = np.ones(1)
    p = C.c_void_p(x.ctypes.data)
    L = _ffi.lib()
    assert L.afar_debug_arithmetic(0, 12, 1, p, p, p) == 1
    assert L.afar_debug_arithmetic(0, -1, 1, p, p, p) == 1
    assert L.afar_debug_arithmetic(0, 0, 1, None, p, p) == 1
