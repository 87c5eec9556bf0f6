"""Division by a value known in advance, as the prefill attention divides its output rows by their sums of weights (b >= 1)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = os.path.join(tmp_path_factory.mktemp("quotient"), "quotient.so")
    subprocess.check_call(["g++", "-O3", "-std=c++17", "-mavx2", "-mfma", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                           os.path.join(HERE, "quotient_check.cpp")])
    lib = C.CDLL(so)
    lib.all_significands.restype = C.c_long
    return lib


def pairs(check, a, b):
    a, b = (np.ascontiguousarray(v, dtype=np.float32) for v in (a, b))
    got, want = np.empty_like(a), np.empty_like(a)
    check.pairs(*(v.ctypes.data_as(C.c_void_p) for v in (a, b, got, want)), C.c_long(a.size))
    return got, want


def test_every_significand_over_divisors_of_the_range(check):
    rng = np.random.default_rng(1)
    edge = np.uint32(0x3F800000) + np.concatenate([np.arange(8), 2 ** 23 - 1 - np.arange(8), 2 ** np.arange(3, 23)]).astype(np.uint32)
    b = np.concatenate([edge.view(np.float32), rng.uniform(1, 2, 60).astype(np.float32), np.float32([3, 5, 7, 10, 1000, 2 ** 20 - 1])])
    assert check.all_significands(b.ctypes.data_as(C.c_void_p), len(b)) == 0


def test_all_exponents(check):
    rng = np.random.default_rng(2)
    n = 1 << 22
    a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-149, 128, n)).astype(np.float32) * rng.choice(np.float32([-1, 1]), n)
    b = np.ldexp(rng.uniform(1, 2, n), rng.integers(0, 21, n)).astype(np.float32)
    got, want = pairs(check, a, b)
    normal = np.abs(a) >= 2.0 ** -100
    assert np.array_equal(got[normal].view(np.int32), want[normal].view(np.int32))
    # the remainder of a smaller one is rounded to a multiple of 2^-149: half of that, twice, before the last rounding
    assert (np.abs(got[~normal].astype(np.float64) - want[~normal]) <= np.maximum(np.spacing(np.abs(want[~normal])), 2.0 ** -149)).all()


def test_zero_infinities_and_nan(check):
    a = np.float32([0, -0.0, np.inf, -np.inf, np.nan, np.finfo(np.float32).max, -np.finfo(np.float32).max])
    for d in (1.0, 1.5, 3.0, 2.0 ** 20):
        got, want = pairs(check, a, np.full_like(a, d))
        assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_newton_step_from_an_approximate_reciprocal(check, ulps):
    """The decode step's division: from a reciprocal that is off by up to two units in the last place (the hardware's by one) the
    quotient is within an ulp and a half, the rounding of r and that of the product."""
    rng = np.random.default_rng(3)
    n = 1 << 22
    a, b = (np.ldexp(rng.uniform(1, 2, n), rng.integers(-30, 31, n)).astype(np.float32) for _ in range(2))
    b[:2 ** 12] = np.float32(1) + np.arange(2 ** 12, dtype=np.float32) * np.float32(2.0 ** -23)     # the ends of a binade
    b[2 ** 12:2 ** 13] = np.float32(2) - np.arange(1, 2 ** 12 + 1, dtype=np.float32) * np.float32(2.0 ** -23)
    out = np.empty_like(a)
    check.newton(*(v.ctypes.data_as(C.c_void_p) for v in (a, b, out)), C.c_long(n), ulps)
    want = a.astype(np.float64) / b.astype(np.float64)
    assert (np.abs(out - want) / np.spacing(np.abs(want).astype(np.float32))).max() <= 1.5
