"""The integer FP64 division (achr.cu_gb300/csrc/achr_div.cuh) where its digits are estimated with an
approximate reciprocal: on the CPU with one that is off by the stated 2^-21 either way, on the GPU with
the instruction the sampler uses.  The operands are test_div.py's; quotients are compared bit for bit."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_div import CSRC, _double

KINDS = ["random", "top", "bottom", "close", "short"]


def _operands(kind, n=1_000_000):
    rng = np.random.default_rng(5)
    top = (1 << 52) - 1
    fa, fb = (rng.integers(0, top + 1, n).astype(np.uint64) for _ in range(2))
    if kind == "top":
        fa = (top - rng.integers(0, 4, n)).astype(np.uint64)
    elif kind == "bottom":
        fb = rng.integers(0, 4, n).astype(np.uint64)
    elif kind == "close":
        fa = (np.clip(fb.astype(np.int64) + rng.integers(-4, 5, n), 0, top)).astype(np.uint64)
    elif kind == "short":
        fb &= np.uint64(0xFFFFF00000000)
        fa &= np.uint64(0xFFFFFFF000000)
    return _double(rng, fa), _double(rng, fb)


def _special():
    v = np.array([0.0, -0.0, -1.0, 5e-324, 1e-310, 2.3e-308, 1.0, 1.7e308, np.inf, np.nan])
    return [np.ascontiguousarray(x.ravel()) for x in np.meshgrid(v, v[3:])]


def _same(got, want):
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


@pytest.mark.parametrize("off", [-1.0, 1.0])
def test_reciprocal_off_by_its_bound(tmp_path, off):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "div.cpp").write_text(r"""
static float off_rcp(float x) { return (float)((1.0 + OFF * 4.76837158203125e-07) / (double)x); }
#define ACHR_DIV_RCP off_rcp
#include "achr_div.cuh"
extern "C" void divide(int n, const double *a, const double *b, double *q) {
    for (int i = 0; i < n; ++i) q[i] = achr::div_rn(a[i], b[i]);
}
""")
    so = tmp_path / "libdiv.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", f"-DOFF={off}", "-I", str(CSRC),
                    str(tmp_path / "div.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    ptr = C.POINTER(C.c_double)
    for kind in KINDS:
        a, b = _operands(kind)
        q = np.empty_like(a)
        lib.divide(len(a), a.ctypes.data_as(ptr), b.ctypes.data_as(ptr), q.ctypes.data_as(ptr))
        with np.errstate(over="ignore", under="ignore"):
            assert _same(q, a / b), kind


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("div") / "libdiv_device.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", str(CSRC), str(Path(__file__).resolve().parent / "cuda" / "div_device.cu"), "-o",
                    str(out)], check=True)
    lib = C.CDLL(str(out))
    ptr = C.POINTER(C.c_double)

    def run(a, b):
        q, want = np.empty_like(a), np.empty_like(a)
        assert lib.div_batch(len(a), *(x.ctypes.data_as(ptr) for x in (a, b, q, want))) == 0
        return q, want
    return run


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS + ["special"])
def test_device_quotients(device, kind):
    a, b = _special() if kind == "special" else _operands(kind)
    q, want = device(a, b)
    assert _same(q, want)
    with np.errstate(all="ignore"):
        assert _same(want, a / b)
