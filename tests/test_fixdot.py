"""The fixed-point stencil sums (csrc/fixdot.cuh), built for the host from the same source,
against exact rational arithmetic.

Bound: the result is rounded once (2^-53 of it, at most 2^-53 n of the largest term) and the
fixed-point terms lose below 2^-55 each, so the error of a sum of n terms is below
(n / 2^53) of its largest term; and over each sample its root mean square is no larger than
that of the float64 multiply-add chain the sum stands in for."""

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
    so = tmp_path_factory.mktemp("fixdot") / "libfixdot.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "fixdot_host.cpp")], check=True)
    dll = ctypes.CDLL(str(so))

    def call(name, x, w):
        x, w = np.ascontiguousarray(x, np.float64), np.ascontiguousarray(w, np.float64)
        out = np.empty(x.shape[0])
        getattr(dll, name)(*(ctypes.c_void_p(a.ctypes.data) for a in (x, w, out)), ctypes.c_long(x.shape[0]))
        return out
    call.dll = dll
    return call


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


KINDS = {"fx_dot10": 10, "fx_dot14": 14, "fx_sum6": 6}


def _sample(rng, kind, rows, spread):
    n = KINDS[kind]
    x = rng.standard_normal((rows, n)) * 2.0 ** rng.uniform(-spread, spread, (rows, n))
    w = rng.standard_normal((rows, n)) * 2.0 ** rng.uniform(-spread / 4, spread / 4, (rows, n))
    return x, (np.sign(w) if kind == "fx_sum6" else w)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("spread", [0, 4, 40, 200])
@pytest.mark.parametrize("cancel", [False, True])
def test_error(lib, kind, spread, cancel):
    n = KINDS[kind]
    x, w = _sample(np.random.default_rng(spread + n), kind, 600, spread)
    if cancel:  # pairs that cancel to a few parts in 1e9
        h = n // 2
        x[:, h:2 * h], w[:, h:2 * h] = x[:, :h] * (1.0 + 1e-9), -w[:, :h]
    got = lib(kind, x, w)
    assert not np.isnan(got).any()
    err, chain = [], []
    for i in range(x.shape[0]):
        terms = [Fraction(a) * Fraction(b) for a, b in zip(x[i], w[i])]
        big, exact, acc = max(map(abs, terms)), sum(terms), 0.0
        for t in terms:
            acc = float(t + Fraction(acc))  # a fused multiply-add chain
        err.append(float(abs(Fraction(got[i]) - exact) / big))
        chain.append(float(abs(Fraction(acc) - exact) / big))
    assert max(err) <= n * 2.0 ** -53
    assert np.sqrt(np.mean(np.square(err))) <= np.sqrt(np.mean(np.square(chain)))


@pytest.mark.parametrize("kind", KINDS)
def test_exact_values(lib, kind):
    """Integers, zeros, subnormal and unused slots are summed exactly; terms that cancel
    exactly give zero."""
    rng = np.random.default_rng(3)
    n = KINDS[kind]
    x = rng.integers(-1000, 1001, (500, n)).astype(np.float64)
    w = rng.integers(-1000, 1001, (500, n)).astype(np.float64)
    if kind == "fx_sum6":
        w = np.where(w < 0, -1.0, 1.0)
    x[::3, n // 2:] = 0.0
    x[::5, 1] = -0.0
    x[::7, 2] = 5e-324
    want = (np.where(np.abs(x) < 1e-300, 0.0, x) * w).sum(1)
    assert np.array_equal(lib(kind, x, w), want)
    x[:, n // 2:2 * (n // 2)] = x[:, :n // 2]
    w[:, n // 2:2 * (n // 2)] = -w[:, :n // 2]
    assert np.array_equal(lib(kind, x + 0.1, w), np.zeros(500))
    assert np.array_equal(lib(kind, np.zeros((4, n)), w[:4]), np.zeros(4))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e-320, 1.7e308])
def test_refused(lib, kind, value):
    """Sums the format cannot hold are handed back to float64."""
    n = KINDS[kind]
    x, w = _sample(np.random.default_rng(5), kind, n, 0)
    if abs(value) < 1.0:
        x[:] = value
    else:
        x[np.arange(n), np.arange(n)] = value
    if value == 1.7e308:
        w = np.sign(w) * 2.0 ** (0 if kind == "fx_sum6" else 40)
        x[:] = value
    assert np.isnan(lib(kind, x, w)).all()


def test_refused_weights(lib):
    x, w = _sample(np.random.default_rng(6), "fx_dot10", 3, 0)
    w[0, 4], w[1, 4], w[2, 4] = np.inf, np.nan, 1e-310
    assert np.isnan(lib("fx_dot10", x, w)).all()


def test_selections(lib):
    """The integer-side selections: x > 0, clamp to [0, 1] (NaN gives 0), float64 order."""
    x = np.array([0.0, -0.0, 5e-324, -5e-324, 1.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), -1.0, 0.3, 1e308,
                  np.inf, -np.inf, np.nan, -np.nan])
    pos, clamp, key, back = np.empty_like(x), np.empty_like(x), np.empty(x.size, np.int64), np.empty_like(x)
    lib.dll.fx_select(_p(x), _p(pos), _p(clamp), _p(key), _p(back), ctypes.c_long(x.size))
    assert np.array_equal(pos, np.where(x > 0.0, x, 0.0)) and not np.signbit(pos).any()
    assert np.array_equal(clamp, np.fmin(np.fmax(x, 0.0), 1.0)) and not np.signbit(clamp).any()
    assert np.array_equal(back.view(np.int64), x.view(np.int64))
    num = ~np.isnan(x)
    a, b = x[num][:, None], x[num][None, :]
    ka, kb = key[num][:, None], key[num][None, :]
    assert np.all((a < b) <= (ka < kb)) and np.all((a > b) <= (ka > kb))
    assert key[x == np.inf][0] < key[np.isnan(x) & ~np.signbit(x)][0]
    assert key[x == -np.inf][0] > key[np.isnan(x) & np.signbit(x)][0]


def test_parts(lib):
    """Positive and negative parts of alternating sums: within a rounding of the exact parts."""
    x, _ = _sample(np.random.default_rng(9), "fx_sum6", 400, 20)
    x[::4, 2] = 0.0
    x[7] = 0.0
    x[8, 0] = np.nan
    x[9, 3] = np.inf
    pos, neg, ok = np.empty(400), np.empty(400), np.empty(400, np.int32)
    lib.dll.fx_parts6(_p(x), _p(pos), _p(neg), _p(ok), ctypes.c_long(400))
    assert list(np.where(ok == 0)[0]) == [8, 9]
    assert pos[7] == 0.0 and neg[7] == 0.0
    for i in np.where(ok)[0]:
        t = [Fraction(v) * (-1) ** j for j, v in enumerate(x[i])]
        big = max(map(abs, t))
        for got, want in ((pos[i], sum(max(v, 0) for v in t)), (neg[i], sum(max(-v, 0) for v in t))):
            assert abs(Fraction(got) - want) <= 6 * Fraction(1, 2 ** 53) * big
