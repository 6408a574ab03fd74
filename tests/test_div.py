"""CPU: the integer FP64 division of the chain kernel (achr.cu_gb300/csrc/achr_div.cuh), compiled here
with the host C++ compiler, equals the hardware's quotient bit for bit: random significands, the
largest and smallest, nearly equal operands, exact quotients, and the operands it hands back."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "achr.cu_gb300" / "csrc"
WRAPPER = r"""
#include "achr_div.cuh"
extern "C" void divide(int n, const double *a, const double *b, double *q) {
    for (int i = 0; i < n; ++i) q[i] = achr::div_rn(a[i], b[i]);
}
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text(WRAPPER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "div.cpp"), "-o",
                    str(d / "libdiv.so")], check=True)
    lib = C.CDLL(str(d / "libdiv.so"))
    ptr = C.POINTER(C.c_double)

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        q = np.empty_like(a)
        lib.divide(len(a), a.ctypes.data_as(ptr), b.ctypes.data_as(ptr), q.ctypes.data_as(ptr))
        return q
    return run


def _double(rng, frac, lo=700, hi=1300):
    exp = rng.integers(lo, hi, len(frac)).astype(np.uint64)
    return ((exp << np.uint64(52)) | frac).view(np.float64)


@pytest.mark.parametrize("kind", ["random", "top", "bottom", "close", "short"])
def test_quotients_equal_the_hardware(divide, kind):
    rng = np.random.default_rng(3)
    n, top = 1_000_000, (1 << 52) - 1
    fa, fb = (rng.integers(0, top + 1, n).astype(np.uint64) for _ in range(2))
    if kind == "top":
        fa = (top - rng.integers(0, 4, n)).astype(np.uint64)
    elif kind == "bottom":
        fb = rng.integers(0, 4, n).astype(np.uint64)
    elif kind == "close":
        fa = (np.clip(fb.astype(np.int64) + rng.integers(-4, 5, n), 0, top)).astype(np.uint64)
    elif kind == "short":  # many exact quotients
        fb &= np.uint64(0xFFFFF00000000)
        fa &= np.uint64(0xFFFFFFF000000)
    a, b = _double(rng, fa), _double(rng, fb)
    with np.errstate(over="ignore", under="ignore"):
        want = a / b
    assert np.array_equal(divide(a, b).view(np.uint64), want.view(np.uint64))


def test_special_operands(divide):
    v = np.array([0.0, -0.0, -1.0, 5e-324, 1e-310, 2.3e-308, 1.0, 1.7e308, np.inf, np.nan])
    a, b = (x.ravel() for x in np.meshgrid(v, v[3:]))
    with np.errstate(all="ignore"):
        want = a / b
    got = divide(a, b)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.uint64), want[ok].view(np.uint64))
