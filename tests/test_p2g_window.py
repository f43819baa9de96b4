"""The P2G window's choice (csrc/ff_window.h), compiled for the host: whatever the
particles' spread, the window fits its shared memory and lies in the domain, up to the
flattest grids that 32-bit face indices allow; on a grid that fits whole it is the
whole spread."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
from conftest import ROOT

SOURCE = """
#include "ff_window.h"
extern "C" int cap() { return P2G_CAP; }
extern "C" void window(const int *q20, const int *q80, const int *n, int count, int *lo, int *w) {
    const int a[3] = {q20[0], q20[1], q20[2]}, b[3] = {q80[0], q80[1], q80[2]}, c[3] = {n[0], n[1], n[2]};
    int l[3], e[3];
    p2g_window(a, b, c, count, l, e);
    for (int q = 0; q < 3; ++q) lo[q] = l[q], w[q] = e[q];
}
"""


@pytest.fixture(scope="module")
def window(tmp_path_factory):
    d = tmp_path_factory.mktemp("window")
    (d / "w.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "tsl_array_n_gb300", "csrc"), str(d / "w.cpp"), "-o", str(d / "w.so")], check=True)
    lib = C.CDLL(str(d / "w.so"))

    def choose(q20, q80, n, count=1 << 30):
        ints = lambda v: (C.c_int * 3)(*[int(x) for x in v])
        lo, w = ints((0, 0, 0)), ints((0, 0, 0))
        lib.window(ints(q20), ints(q80), ints(n), count, lo, w)
        return list(lo), list(w)

    return choose, lib.cap()


FLAT = [(20000, 20000, 1), (28000, 28000, 1), (30000, 30000, 1), (32700, 32700, 1), (1, 32700, 32700), (32700, 1, 32700),
        (1289, 1289, 1289), ((1 << 29) - 10, 1, 1), (26000, 26000, 2)]


@pytest.mark.parametrize("n", FLAT + [(256, 128, 128), (7, 5, 3), (1, 1, 1)])
@pytest.mark.parametrize("spread", ["whole domain", "scattered samples", "a row"])
def test_window_fits(window, n, spread):
    choose, cap = window
    assert np.prod([x + 1 for x in n], dtype=object) < 2 ** 31      # grids the solver takes
    rng = np.random.default_rng(sum(n))
    for _ in range(200):
        if spread == "whole domain":
            q20, q80 = [0, 0, 0], [x - 1 for x in n]
        elif spread == "scattered samples":
            s = np.sort(np.stack([rng.integers(0, x, 32) for x in n]), axis=1)
            q20, q80 = s[:, 6], s[:, 25]
        else:
            at = [int(rng.integers(0, x)) for x in n]
            q20, q80 = [0, at[1], at[2]], [n[0] - 1, at[1], at[2]]
        lo, w = choose(q20, q80, n)
        assert (w[0] + 2) * (w[1] + 2) * (w[2] + 2) <= cap
        for b in range(3):
            assert w[b] >= 1 and lo[b] >= 0 and lo[b] + w[b] <= n[b]


def test_window_of_a_small_domain_is_its_spread(window):
    choose, _ = window
    assert choose((0, 0, 0), (6, 4, 2), (7, 5, 3)) == ([0, 0, 0], [7, 5, 3])
    assert choose((10, 3, 3), (13, 3, 3), (64, 8, 8)) == ([9, 3, 3], [6, 1, 1])


def test_no_window_for_a_run_spread_thinner_than_its_additions(window):
    choose, cap = window
    whole = ((0, 0, 0), (255, 127, 127), (256, 128, 128))
    assert choose(*whole, count=4096)[1] == [0, 0, 0]
    row = ((0, 3, 3), (255, 4, 3), (256, 128, 128))     # two rows: 258 x 6 x 5 faces or fewer
    lo, w = choose(*row, count=4096)
    assert min(w) >= 1 and (w[0] + 2) * (w[1] + 2) * (w[2] + 2) <= cap
    assert choose((2, 2, 2), (2, 2, 2), (8, 8, 8), count=1)[1] == [0, 0, 0]
    args = ((10, 3, 0), (13, 3, 0), (64, 8, 1))         # 8 x 3 x 3 faces: nine particles' additions
    assert choose(*args, count=8)[1] == [0, 0, 0] and choose(*args, count=9)[1] == [6, 1, 1]
    for n in FLAT:
        for count in (1, 512, 4096):
            w = choose((0, 0, 0), [x - 1 for x in n], n, count=count)[1]
            assert w == [0, 0, 0] or np.prod([x + 2 for x in w]) <= min(cap, 8 * count)
