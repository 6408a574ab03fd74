"""CPU: the configuration a launch of few chains takes (achr.cu_gb300/csrc/achr_chain_rule.h, compiled here with
the host C++ compiler): more threads per chain up to 16 warps on an SM, for models that reproject through
the residual too where the configuration can take the default's turns of z."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "achr.cu_gb300" / "csrc"
WRAPPER = r"""
#include "achr_chain_rule.h"
using namespace achr;
static int code(const ChainCfg *c) { return c ? c->bd * 100 + c->ept : 0; }
extern "C" int dflt(int n, int scratch) { return code(find_cfg(n, 0, scratch)); }
extern "C" int few(int n, int max_np, int m, int scratch, int turn, int per_sm) {
    return code(few_chains_cfg(find_cfg(n, 0, scratch), n, max_np, m, scratch, turn, per_sm));
}
extern "C" int room(int c, int m) { return 2 * (cfg_scratch({c / 100, c % 100, false}) - m); }
extern "C" int turns(int c, int m) { return residual_z_rows(m, cfg_scratch({c / 100, c % 100, false})); }
extern "C" int alloc(int n, int most) { return chain_alloc_length(n, most); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("chain_rule")
    (d / "rule.cpp").write_text(WRAPPER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rule.cpp"),
                    "-o", str(d / "librule.so")], check=True)
    return C.CDLL(str(d / "librule.so"))


def _np(c):
    return (c // 100) * (c % 100)


@pytest.mark.parametrize("n,m,turn,per_sm,want", [
    (7440, 5063, 2162, 1, 51216), (7440, 5063, 2162, 2, 25630),  # three turns of z in either
    (7440, 7000, 100, 1, 51216), (7440, 7400, 1600, 1, 25630),   # 792 doubles beside 7400 residuals: 1584 rows
    (1060, 911, 911, 1, 51204), (1060, 911, 911, 2, 25608), (1060, 911, 911, 9, 6420),
    (250, 190, 190, 1, 12804), (250, 190, 190, 7, 6404), (250, 190, 190, 9, 3208),
])
def test_residual_form(lib, n, m, turn, per_sm, want):
    assert lib.few(n, lib.alloc(n, 16384), m, m if n < 7000 else 6000, turn, per_sm) == want


def test_any_size(lib):
    for n in [*range(1, 8193, 41), 128, 129, 256, 257, 1280, 1281, 3840, 3841, 6656, 6657, 7680, 7681, 8192]:
        d = lib.dflt(n, 0)
        for max_np in {lib.alloc(n, 16384), _np(d)}:
            for m in (1, n // 2, n):
                for turn in {0, m, max(1, m // 3)}:
                    for per_sm in (1, 2, 3, 5, 8, 16, 17):
                        c = lib.few(n, max_np, m, 0, turn, per_sm)
                        assert n <= _np(c) <= max_np
                        if c != d:
                            assert c // 100 > d // 100 and per_sm * (c // 3200) <= 16
                            assert turn == 0 or turn == m or lib.room(c, m) >= turn


def test_room_without_allocation(lib):
    """achr_sample_noalloc's arrays hold 8192 reactions at most: what fits them is what a context would take."""
    for n in [*range(1, 8193, 41), 1060, 2500, 7680, 8192]:
        for per_sm in (1, 2, 4):
            want = lib.few(n, lib.alloc(n, 16384), 0, 0, 0, per_sm)
            assert _np(want) > 8192 or lib.few(n, lib.alloc(n, 8192), 0, 0, 0, per_sm) == want
    assert lib.few(1060, lib.alloc(1060, 8192), 0, 0, 0, 1) == 51204
