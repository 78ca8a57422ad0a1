"""The reciprocals, quotients and roots of the pointwise physics (recip.cuh) on
the GPU, through the check hook of include/dgb200_check.h."""
import ctypes

import numpy as np
import pytest

import dgpr_b200 as dg

pytestmark = pytest.mark.gpu

_dp = ctypes.POINTER(ctypes.c_double)
RCP, QUOT, SQRT, RCP_ROOT, RSQRT = range(5)
DOUBLE, FLOAT, PAIR = range(3)


def call(f, kind, a, b):
    fn = dg.lib().dgb_check_arithmetic
    fn.restype, fn.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, _dp, _dp, _dp]
    y = np.zeros(2 * a.size)
    assert fn(f, kind, a.size, *(v.ctypes.data_as(_dp) for v in (a, b, y))) == 0
    return y[: a.size], y[a.size:]


def values(rng, n, lo, hi, dtype):
    """Spread over lo .. hi in their logarithm, and around the powers of two and their roots."""
    v = np.exp(rng.uniform(np.log(lo), np.log(hi), n)).astype(dtype)
    e = np.exp2(np.arange(np.ceil(np.log2(lo)) + 1, np.floor(np.log2(hi)))).astype(dtype)
    e = np.concatenate([e, np.sqrt(e), e * dtype(1.5)])
    near = [e]
    for _ in range(3):
        near.append(np.nextafter(near[-1], dtype(np.inf)))
    down = [e]
    for _ in range(3):
        down.append(np.nextafter(down[-1], dtype(0)))
    return np.concatenate([v, *near, *down]).astype(np.float64)


def ulps(y, want, dtype):
    """Distance of y from the wider want in units of the last place of want."""
    return np.abs((y.astype(want.dtype) - want) / np.spacing(np.abs(want).astype(dtype)).astype(want.dtype))


@pytest.mark.parametrize("f", [RCP, QUOT, SQRT, RCP_ROOT])
def test_double_rounds_as_the_operators(f):
    """Over 1e-17 .. 1e17, against 80-bit arithmetic (2^-11 of a unit in the
    last place): the last step of each leaves its result some 2^-39 of a unit
    from the exact value before it rounds, so within 0.5 + 2^-10 units, as the
    operator; 1 / sqrt is that of the rounded root, each side of its own (the
    root of 1 - 2^-53 is 2^-56 units from a tie, either neighbour of which is
    within the bar)."""
    rng = np.random.default_rng(f)
    a = values(rng, 1 << 20, 1e-17, 1e17, np.float64)
    b = rng.permutation(a)
    y, op = call(f, DOUBLE, a, b)
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    for v, root in zip((y, op), call(SQRT, DOUBLE, a, b)):
        want = {RCP: 1 / A, QUOT: A / B, SQRT: np.sqrt(A), RCP_ROOT: 1 / root.astype(np.longdouble)}[f]
        assert ulps(v, want, np.float64).max() <= 0.5 + 2.0 ** -10


@pytest.mark.parametrize("kind", [FLOAT, PAIR], ids=["float", "pair"])
@pytest.mark.parametrize("f", [RCP, QUOT, SQRT, RCP_ROOT])
def test_float_rounds_as_the_operators(f, kind):
    """Over 2e-9 .. 5e8, against float64: within 0.5 units and the 2^-20 that
    the refinement leaves; both lanes of a pair."""
    rng = np.random.default_rng(f)
    a = values(rng, 1 << 20, 2e-9, 5e8, np.float32)
    b = rng.permutation(a)
    y, second = call(f, kind, a, b)
    root = np.sqrt(a).astype(np.float32).astype(np.float64)
    want = {RCP: 1 / a, QUOT: a / b, SQRT: np.sqrt(a), RCP_ROOT: 1 / root}[f]
    for v in (y, second):
        assert ulps(v, want, np.float32).max() <= 0.5 + 2.0 ** -20


def test_reciprocal_root_that_they_start_from():
    """1.5 units in FP64 (the product x y rounds once, which the step halves,
    and the step itself) and in FP32."""
    rng = np.random.default_rng(9)
    a = values(rng, 1 << 18, 1e-17, 1e17, np.float64)
    assert ulps(call(RSQRT, DOUBLE, a, a)[0], 1 / np.sqrt(a.astype(np.longdouble)), np.float64).max() <= 1.5
    a = values(rng, 1 << 18, 2e-9, 5e8, np.float32)
    for kind in (FLOAT, PAIR):
        assert ulps(call(RSQRT, kind, a, a)[0], 1 / np.sqrt(a), np.float32).max() <= 1.5
