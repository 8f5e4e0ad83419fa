"""The steps' arithmetic in float pairs, function by function on the device, against extended precision: reciprocals, limited
slopes, differences and upwind values of the FP64 transport within the bounds that their comments state, and
the FP32 march's quotients against IEEE division.
"""
import ctypes

import numpy as np
import pytest

from cudaprotoplanetarydisks_gb300 import _capi

pytestmark = pytest.mark.gpu
RCP, RSQRT, JOIN, LIMITER, LIMITER_SCALED, DIFF, STAR, QUOTIENT, MISMATCHES = range(9)
N = 1 << 18
L = np.longdouble


def run(which, *cols):
    x = np.zeros((len(cols[0]), 4))
    for k, v in enumerate(cols):
        x[:, k] = v
    out, p = np.empty(len(x)), ctypes.POINTER(ctypes.c_double)
    assert _capi.load().fargo_pair_selftest(which, x.ctypes.data_as(p), len(x), out.ctypes.data_as(p)) == 0
    return out


def numbers(rng, lo, hi, n=N):
    return rng.choice([-1.0, 1.0], n) * (1 + rng.random(n)) * 2.0 ** rng.integers(lo, hi, n)


def worst(got, want):
    return float(np.max(np.abs((got.astype(L) - want) / want)))


def test_reciprocals_are_within_an_ulp():
    rng = np.random.default_rng(1)
    for lo, hi in ((-20, 20), (-499, 500), (-1000, 1000)):
        a = numbers(rng, lo, hi)
        want = 1 / a.astype(L)
        assert (np.abs(run(RCP, a).astype(L) - want) <= np.spacing(np.abs(want.astype(float)))).all()
        a = np.abs(a)
        want = 1 / np.sqrt(a.astype(L))
        assert (np.abs(run(RSQRT, a).astype(L) - want) <= np.spacing(want.astype(float))).all()


def test_a_double_from_two_floats():
    rng = np.random.default_rng(2)
    a = numbers(rng, -60, 60).astype(np.float32)
    b = a * (2.0 ** -23 * rng.uniform(-2, 2, N)).astype(np.float32)
    assert worst(run(JOIN, a, b), a.astype(L) + b.astype(L)) <= 2.0 ** -46


# operands of one magnitude, of some, at the ends of what the pairs take, and beyond it
@pytest.mark.parametrize("spread", [0, 3, 19, 29, 60, 400])
@pytest.mark.parametrize("at", [-300, -30, 0, 30, 300])
def test_limiter_fractions(at, spread):
    rng = np.random.default_rng(1000 * spread + at + 500)
    s = rng.choice([-1.0, 1.0], N)
    a = s * np.abs(numbers(rng, at, at + 1))
    b = s * np.abs(numbers(rng, at - spread, at + spread + 1))
    c, rho = numbers(rng, -40, 0), np.abs(numbers(rng, -9, 9))
    al, bl, cl, rl = (v.astype(L) for v in (a, b, c, rho))
    assert worst(run(LIMITER, a, b, c), cl * bl / (al + bl)) <= 2.0 ** -43
    assert worst(run(LIMITER_SCALED, a, b, c, rho), cl * rl * bl / (al + rl * bl)) <= 2.0 ** -42


@pytest.mark.parametrize("apart", [0, 1, 8, 24, 40, 53])
def test_differences(apart):
    rng = np.random.default_rng(apart)
    a = numbers(rng, -29, 40)
    b = a * (1 + 2.0 ** -apart * rng.uniform(-0.999, 1, N))
    b[:100] = a[:100]
    b[100:200] = 0.0
    got, want = run(DIFF, a, b), a.astype(L) - b.astype(L)
    assert (np.abs(got.astype(L) - want) <= 2.0 ** -45 * np.abs(want)).all()
    out = np.array([2.0 ** -41, 1e-300, 5e-324, 2.0 ** 101, np.inf, np.nan])
    assert np.isnan(run(DIFF, out, np.ones(6))).all() and np.isnan(run(DIFF, np.ones(6), out)).all()


@pytest.mark.parametrize("apart", [0, 2, 12, 30, 45])
def test_upwind_values(apart):
    rng = np.random.default_rng(apart)
    b = numbers(rng, -38, 38)
    x, y = (b * 2.0 ** -apart * rng.uniform(-0.5, 0.5, N) for _ in range(2))
    a, d, c = b - y, b + x, numbers(rng, -30, 0)
    al, bl, cl, dl = (v.astype(L) for v in (a, b, c, d))
    xl, yl = dl - bl, bl - al
    with np.errstate(invalid="ignore", divide="ignore"):
        slope = np.where(xl * yl > 0, cl * xl * yl / (xl + yl), 0)
    # the slope's part (dropped below 2^-100) and the rounding of the sum
    bound = 2.0 ** -42 * np.abs(slope) + 2.0 ** -100 + np.spacing(np.abs(b) + np.abs(slope.astype(float))) / 2
    assert (np.abs(run(STAR, a, b, c, d).astype(L) - (bl + slope)) <= bound).all()


def test_fp32_quotients_are_ieee():
    assert run(MISMATCHES, np.full(N, 7.0)).sum() == 0  # 2^30 pairs
    # all significands of the divisor against numerators beside the quotient's midpoints
    b = (np.arange(1 << 18, dtype=np.float64) * 32 + 2 ** 23 + 31) / 2 ** 23
    for m in (1.0, 1.0 + 2.0 ** -23, 1.5, 2 - 2.0 ** -23):
        b32 = b.astype(np.float32)
        a = (b32.astype(np.float64) * (m + 2.0 ** -24)).astype(np.float32)
        assert np.array_equal(run(QUOTIENT, a, b32).astype(np.float32), a / b32)
    zeros = run(QUOTIENT, np.array([0.0, 0.0]), np.array([3.0, -2.0 ** -50]))
    assert np.array_equal(zeros, [0.0, 0.0])
