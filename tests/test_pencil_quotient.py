"""The quotients of the pressure solve along grid lines against the division, on the CPU.

Its sweeps multiply by a pivot's reciprocal where that gives the correctly rounded quotient, and leave
the rest to the division: every quotient they accept equals the division's, no tolerance.  The pairs
cover all magnitudes, exact quotients, quotients on the tie between two subnormals, the borders of
the normal range, zeros and infinities.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("quotient") / "quotient_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-o", out,
                    os.path.join(HERE, "native", "quotient_host.cpp")], check=True)
    return C.CDLL(out)


def _count(lib, s, d):
    s, d = np.broadcast_arrays(s, d)
    s, d = np.ascontiguousarray(s), np.ascontiguousarray(d)
    out = (C.c_int64 * 3)()
    fn = lib.rfh_quotients32 if s.dtype == np.float32 else lib.rfh_quotients64
    fn(s.ctypes.data_as(C.c_void_p), d.ctypes.data_as(C.c_void_p), C.c_int64(s.size), out)
    accepted, differ, first = out
    assert differ == 0, f"{differ} of {accepted} differ, first {s.flat[first]!r} / {d.flat[first]!r}"
    return accepted / s.size


def _random(rng, n, dtype, lo, hi):
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
    return x.astype(dtype)


def test_fp32_quotients_of_all_magnitudes(lib):
    rng = np.random.default_rng(1)
    n = 2_000_000
    with np.errstate(over="ignore"):
        # pivots are above 2.2e-16 in magnitude
        assert _count(lib, _random(rng, n, np.float32, -149, 128), _random(rng, n, np.float32, -52, 128)) > 0.99
        # quotients around the smallest normal number and among the subnormals
        d = _random(rng, n, np.float32, -20, 20)
        s = (d.astype(np.float64) * _random(rng, n, np.float64, -152, -124)).astype(np.float32)
        assert _count(lib, s, d) > 0.99


def test_fp32_quotients_on_ties_of_subnormals(lib):
    rng = np.random.default_rng(2)
    n = 400_000
    # s = d (m + 1/2) 2^-149 exactly: m below 2^12 and d of at most 11 bits
    m = rng.integers(0, 1 << 12, n)
    d = rng.integers(1, 1 << 11, n).astype(np.float64)
    e = rng.integers(2, 30, n)
    s = np.ldexp(d * (2 * m + 1), -150 + e)
    s32, d32 = s.astype(np.float32), np.ldexp(d, e).astype(np.float32)
    assert np.array_equal(s32.astype(np.float64), s)
    _count(lib, s32, d32)
    _count(lib, -s32, d32)
    # the tie between the largest subnormal and the smallest normal number, and those next to zero
    for q in (2 * ((1 << 23) - 1) + 1, 1, 3):
        p = np.ldexp(np.float64(q), -150)
        for dd in (2.0, 4.0, 1024.0):
            _count(lib, np.full(4, p * dd, np.float32), np.full(4, dd, np.float32))


def test_fp64_quotients_of_all_magnitudes(lib):
    rng = np.random.default_rng(3)
    n = 2_000_000
    assert _count(lib, _random(rng, n, np.float64, -800, 800), _random(rng, n, np.float64, -90, 90)) > 0.99
    with np.errstate(over="ignore"):
        _count(lib, _random(rng, n, np.float64, -1074, 1024), _random(rng, n, np.float64, -400, 400))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_exact_quotients_zeros_and_infinities(lib, dtype):
    rng = np.random.default_rng(4)
    d = rng.integers(1, 4000, 200_000).astype(dtype)
    _count(lib, (d * rng.integers(-4000, 4000, d.size)).astype(dtype), d)
    for s in (0.0, -0.0, np.inf, -np.inf, np.nan):
        _count(lib, np.array([s], dtype), np.array([3.0, -0.7, 1e-9, 1e9], dtype))
