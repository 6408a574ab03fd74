"""CPU: which runs are deferred (achr.cu_gb300/csrc/achr_defer_rule.h), and that buffers a capture has seen
outlive their replacements (achr_kept.h), compiled here with the host C++ compiler."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "achr.cu_gb300" / "csrc"
WRAPPER = r"""
#include "achr_defer_rule.h"
#include "achr_kept.h"
extern "C" int rule(int selected, int asked, double chains, double nd, int capturing) {
    int short_from = 0;
    return achr::defer_choose(achr::defer_use(selected, asked, chains, nd), capturing, (int)chains, short_from,
                              [] { return achr::DeferBuffers::kReady; }).deferred;
}
// A context's runs one after another: chains of each, and what asking for its buffers would give ('r' ready,
// 'm' no memory, 'x' another failure).  What each did: 'd' deferred, 'k' in the kernel, 'e' an error; in
// upper case if the buffers were asked for.
extern "C" void runs(int n, const int *chains, const char *buffers, char *did) {
    int short_from = 0;
    for (int i = 0; i < n; ++i) {
        bool asked = false;
        const achr::DeferChoice c = achr::defer_choose(achr::DeferUse::kMay, false, chains[i], short_from, [&] {
            asked = true;
            return buffers[i] == 'r'   ? achr::DeferBuffers::kReady
                   : buffers[i] == 'm' ? achr::DeferBuffers::kNoMemory
                                       : achr::DeferBuffers::kFailed;
        });
        did[i] = (c.failed ? 'e' : c.deferred ? 'd' : 'k') - (asked ? 32 : 0);
    }
}
static int alive;
struct Buf {
    Buf() { ++alive; }
    ~Buf() { --alive; }
};
// steps: 'g' grows (a new buffer), 'f' fails to grow, 'c' captures; returns the buffers still allocated,
// and 1000 more where the owner's end leaves any behind
extern "C" int kept(const char *steps) {
    alive = 0;
    int end;
    {
        achr::Kept<Buf> k;
        for (; *steps; ++steps) {
            if (*steps == 'c') k.captured();
            if (*steps == 'g' || *steps == 'f') k.retire();
            if (*steps == 'g') k.replace(std::unique_ptr<Buf>(new Buf()));
        }
        end = alive;
    }
    return end + (alive ? 1000 : 0);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(WRAPPER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rule.cpp"),
                    "-o", str(d / "librule.so")], check=True)
    so = C.CDLL(str(d / "librule.so"))
    so.rule.argtypes = [C.c_int, C.c_int, C.c_double, C.c_double, C.c_int]
    so.runs.argtypes = [C.c_int, C.POINTER(C.c_int), C.c_char_p, C.c_char_p]
    so.kept.argtypes = [C.c_char_p]
    return so


@pytest.mark.parametrize("selected,asked,chains,nd,capturing,deferred", [
    (0, 0, 1e6, 1e6, 0, 0),       # the model or the options do not allow it
    (1, 0, 1e4, 1999.0, 0, 0), (1, 0, 1e4, 2000.0, 0, 1),  # the line of chains x n d
    (1, 0, 1.0, 2.5e5, 0, 1), (1, 0, 1.0, 2.49e5, 0, 0),   # the line of n d
    (1, 0, 1e4, 1e5, 1, 0),       # a capture stays in the kernel where that is a choice
    (1, 0, 1.0, 2.5e5, 1, 1), (1, 1, 1.0, 1.0, 1, 1), (1, 1, 1.0, 1.0, 0, 1),
])
def test_line(lib, selected, asked, chains, nd, capturing, deferred):
    assert lib.rule(selected, asked, chains, nd, capturing) == deferred


@pytest.mark.parametrize("chains,buffers,did", [
    ([100, 100], "rr", "DD"),
    ([100, 100, 100], "mrr", "Kkk"),            # short once: every later run of that size stays in the kernel
    ([100, 200, 50, 100], "mrrr", "KkDk"),      # and the larger ones; smaller ones are asked for
    ([100, 50, 70, 20], "mmrr", "KKkD"),
    ([100, 100], "xr", "ED"),                   # any other failure is the call's, and not remembered
])
def test_memory_short(lib, chains, buffers, did):
    out = C.create_string_buffer(len(chains) + 1)
    lib.runs(len(chains), (C.c_int * len(chains))(*chains), buffers.encode(), out)
    assert out.value.decode() == did


@pytest.mark.parametrize("steps,left", [("", 0), ("g", 1), ("gg", 1), ("ggg", 1), ("c", 0), ("gc", 1), ("gcg", 2),
                                        ("gcgg", 2), ("gcgcg", 3), ("gccg", 2), ("gf", 0), ("gcf", 1), ("gcfg", 2),
                                        ("gcfcg", 2), ("gcggcf", 2)])
def test_captured_buffers_are_kept(lib, steps, left):
    assert lib.kept(steps.encode()) == left
