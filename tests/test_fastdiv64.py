"""The kernels' float64 quotient and reciprocal (csrc/fastdiv64.cuh), built for the host from
the same source, against IEEE division: the same bits on every sampled argument, with the
float32 seed exact or an ulp off either way, and on every argument that takes the
compiler's division; next to a tie (1 / (1 - 2^-53)) within half an ulp and 2^-30 of one."""

from __future__ import annotations

import ctypes
import pathlib
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    so = tmp_path_factory.mktemp("fastdiv") / "libfastdiv.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "fastdiv64_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def _divide(lib, a, b, ulps=0):
    out = np.empty_like(a)
    lib.quotients(_p(a), _p(b), _p(out), ctypes.c_long(a.size), ctypes.c_int(ulps))
    return out


@pytest.mark.parametrize("ulps", [-1, 0, 1])
@pytest.mark.parametrize("spread", [0.5, 8.0, 65.0])
def test_quotient_is_the_rounded_one(lib, ulps, spread):
    rng = np.random.default_rng(int(spread) + 2 + ulps)
    b = np.exp2(rng.uniform(-1.4 * spread, spread, 300_000))
    a = rng.standard_normal(b.size) * np.exp2(rng.uniform(-spread, spread, b.size))
    assert np.array_equal(_divide(lib, a, b, ulps), a / b)


def test_edges(lib):
    one = np.nextafter(1.0, 2.0)
    b = np.array([1.0, one, np.nextafter(1.0, 0.0), 2.0, np.nextafter(2.0, 1.0), 3.0, 1.0 + 2.0 ** -24,
                  2.0 ** -100, np.nextafter(2.0 ** -100, 0.0), 2.0 ** 70, np.nextafter(2.0 ** 70, 0.0), 1e-20, 0.0, -0.0, -3.0,
                  5e-324, 1e-310, np.inf, -np.inf, np.nan, 1e300])
    a = np.array([0.0, -0.0, 1.0, -1.0, 3.0, one, 2.0 ** -600, np.nextafter(2.0 ** -600, 0.0), 2.0 ** 799, 2.0 ** 801,
                  5e-324, np.inf, np.nan, 1e308])
    aa, bb = (np.ascontiguousarray(x.ravel()) for x in np.meshgrid(a, b))
    with np.errstate(all="ignore"):
        want = aa / bb
        inv = 1.0 / b
    got = _divide(lib, aa, bb)
    for x, y, g, w in zip(aa, bb, got, want):
        if np.isnan(w) or np.isinf(w) or w == 0.0 or g == w:
            assert np.array_equal(g, w, equal_nan=True) and (np.isnan(w) or np.signbit(g) == np.signbit(w)), (x, y)
        else:  # a quotient within 2^-80 of the middle of two float64 values may round either way
            off = abs(Fraction(g) - Fraction(x) / Fraction(y))
            assert off <= Fraction(np.spacing(abs(g))) * (Fraction(1, 2) + Fraction(1, 2 ** 30)), (x, y)
    out = np.empty_like(b)
    lib.reciprocals(_p(b), _p(out), ctypes.c_long(b.size))
    same = np.isnan(inv) | np.isinf(inv) | (np.abs(b - 1.0) > 1e-15) & (np.abs(b - 2.0) > 1e-15) & (b < 2.0 ** 69)
    assert np.array_equal(out[same], inv[same], equal_nan=True)
    assert np.all(np.abs(out[~same] - inv[~same]) <= np.spacing(inv[~same]))


def test_reciprocal(lib):
    b = np.exp2(np.random.default_rng(1).uniform(-99, 69, 300_000))
    out = np.empty_like(b)
    lib.reciprocals(_p(b), _p(out), ctypes.c_long(b.size))
    assert np.array_equal(out, 1.0 / b)
