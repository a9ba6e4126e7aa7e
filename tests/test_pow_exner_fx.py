"""pow_exner_fx (csrc/pow_exner_fx.cuh), the float64 step's Exner-function pow on the integer
pipes, built for the host from the same source: correctly rounded against 50-digit decimal
arithmetic, and pow_exner's bits but for the one case in 2^18 that either may round the other
way next to a boundary (bound: 2^-16 of the samples)."""

from __future__ import annotations

import ctypes
import pathlib
import shutil
import subprocess
import sys
from decimal import Decimal, localcontext

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "mpas_dycore_pytorch_gb300" / "csrc"
RCV = 287.0 / (1004.5 - 287.0)
RANGES = [(0.01, 2.0, RCV), (1e-5, 1e5, 0.37), (0.5, 1.5, 3.5), (0.9, 1.1, -2.75), (1e-300, 1e300, 0.9),
          (0.999, 1.001, 15.0), (0.2, 1.2, 1e-6)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    so = tmp_path_factory.mktemp("powfx") / "libpowfx.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "pow_exner_fx_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


def _call(fn, x, y):
    x = np.ascontiguousarray(x, np.float64)
    y = np.ascontiguousarray(np.broadcast_to(np.float64(y), x.shape))
    out = np.empty_like(x)
    fn(*(ctypes.c_void_p(a.ctypes.data) for a in (x, y, out)), ctypes.c_long(x.size))
    return out


def _sample(rng, lo, hi, n):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), n)) if hi / lo > 1e3 else rng.uniform(lo, hi, n)


def test_tables_are_generated_from_the_script():
    r = subprocess.run([sys.executable, str(CSRC / "gen_pow_fx_tables.py"), "--check"])
    assert r.returncode == 0, "pow_fx_tables.inc differs from gen_pow_fx_tables.py's output"


@pytest.mark.parametrize("lo,hi,y", RANGES)
def test_correctly_rounded(lib, lo, hi, y):
    x = _sample(np.random.default_rng(7), lo, hi, 400)
    got = _call(lib.pow_fx_many, x, y)
    with localcontext() as ctx:
        ctx.prec = 50
        want = np.array([float((Decimal(float(v)).ln() * Decimal(float(y))).exp()) for v in x])
    assert np.array_equal(got, want), int((got != want).sum())


@pytest.mark.parametrize("lo,hi,y", RANGES)
def test_agrees_with_pow_exner(lib, lo, hi, y):
    n = 1 << 20
    x = _sample(np.random.default_rng(11), lo, hi, n)
    edges = 1.0 + np.arange(1025) / 1024.0  # where the table's row changes
    x[:4096] = np.concatenate([edges, np.nextafter(edges, 0), np.nextafter(edges, 4), 0.5 * edges])[:4096]
    got, ref = _call(lib.pow_fx_many, x, y), _call(lib.pow_dd_many, x, y)
    diff = got != ref
    assert diff.sum() <= n >> 16, int(diff.sum())
    assert np.all(np.abs(got - ref) <= np.spacing(ref))


def test_exact_cases_and_fallbacks(lib):
    x = np.array([1.0, 4.0, 0.25, 2.0, 0.0, -2.0, np.inf, 1e-310, 3.0, np.nan, 1.5, 1.5, 0.7, 1e308, 1e-308, 16.0])
    y = np.array([RCV, 0.5, 0.5, 10.0, RCV, 2.0, 0.5, 0.5, 800.0, RCV, np.nan, 0.0, -np.inf, 3.0, 3.0, -1.25])
    assert np.array_equal(_call(lib.pow_fx_many, x, y), _call(lib.pow_dd_many, x, y), equal_nan=True)
