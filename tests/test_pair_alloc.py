"""Two arrays, both or neither (csrc/ff_pairalloc.h), compiled for the host with an
allocator whose n-th call fails: nothing is left allocated and no pointer stays behind."""
import ctypes as C
import os
import subprocess

import pytest
from conftest import ROOT

SOURCE = """
#include "ff_pairalloc.h"
#include <cstdlib>
// returns the blocks left allocated after the call; got: whether it says both are there,
// second: whether a second try, with an allocator that works, gets both
extern "C" int try_both(int failing, int *got, int *null, int *second) {
    int calls = 0, live = 0;
    void *a = (void *)8, *b = (void *)8;
    auto alloc = [&](void **p, size_t n) {
        *p = nullptr;
        if (++calls == failing) return -3;
        *p = std::malloc(n);
        ++live;
        return 0;
    };
    auto release = [&](void *p) {
        if (p) --live;
        std::free(p);
    };
    *got = alloc_both(&a, 32, &b, 16, alloc, release);
    *null = !a && !b;
    const int left = live;
    if (!*got) *second = alloc_both(&a, 32, &b, 16, alloc, release) && live == left + 2;
    release(a);
    release(b);
    return left;
}
"""


@pytest.mark.parametrize("failing,left", [(0, 2), (1, 0), (2, 0)])
def test_both_or_neither(tmp_path, failing, left):
    (tmp_path / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tsl_array_n_gb300", "csrc"),
                    str(tmp_path / "a.cpp"), "-o", str(tmp_path / "a.so")], check=True)
    got, null, second = C.c_int(), C.c_int(), C.c_int(1)
    n = C.CDLL(str(tmp_path / "a.so")).try_both(failing, C.byref(got), C.byref(null), C.byref(second))
    assert n == left and got.value == (failing == 0) and null.value == (failing != 0) and second.value == 1
