"""Growth of the page-locked staging buffer over a fake allocator (no GPU)."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "solvix_b200", "csrc")

SOURCE = r"""
#include "svx_pinned.h"
static unsigned long long room, held, asked, last;
struct Fake {  // refuses what the host has no room for
    static void* alloc(size_t n) {
        ++asked;
        if (n > room) return nullptr;
        held = last = n;
        return &held;
    }
    static void free(void*) { held = 0; }
};
static svx::PinnedBufferT<Fake>* b;
extern "C" void fresh(unsigned long long host) { b = new svx::PinnedBufferT<Fake>; room = host; held = asked = 0; }
extern "C" void limit(unsigned long long n) { b->limit = n; }
extern "C" int get(unsigned long long n) { return b->try_get(n) != nullptr; }
extern "C" unsigned long long now_held() { return held; }
extern "C" unsigned long long times_asked() { return asked; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pinned")
    (d / "p.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "p.cpp"),
                    "-o", str(d / "p.so")], check=True)
    lib = C.CDLL(str(d / "p.so"))
    for f in (lib.fresh, lib.limit, lib.get):
        f.argtypes = [C.c_ulonglong]
    lib.now_held.restype = lib.times_asked.restype = C.c_ulonglong
    return lib


MB, GB = 1 << 20, 1 << 30


def test_large_sizes_take_what_they_ask_for(lib):
    lib.fresh(6 * GB)
    assert lib.get(5 * GB) and lib.now_held() == 5 * GB
    lib.fresh(6 * GB)
    assert lib.get(256 * MB + 1) and lib.now_held() == 256 * MB + 1


def test_a_refused_doubled_size_is_asked_for_exactly(lib):
    lib.fresh(150 * MB)
    assert lib.get(140 * MB) and lib.now_held() == 140 * MB
    assert lib.get(100 * MB) and lib.times_asked() == 2


def test_small_sizes_double_and_are_kept(lib):
    lib.fresh(GB)
    for n in (1, 5, MB, 3 * MB, 4 * MB, 2 * MB):
        assert lib.get(n)
    assert lib.now_held() == 4 * MB and lib.times_asked() == 2


def test_refusal_is_reported_and_not_for_good(lib):
    lib.fresh(10 * MB)
    assert not lib.get(64 * MB) and lib.now_held() == 0
    assert lib.get(8 * MB)
    lib.limit(MB)
    assert not lib.get(2 * MB) and lib.get(MB)
