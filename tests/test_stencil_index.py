"""The kernels' index tests of a 3x3x3 stencil (csrc/mpm_stencil.h), built with
the host compiler at several optimisation levels: exact against unbounded
integers for every kind of cell, the saturated ones (a coordinate beyond 2^31
or an infinity) among them."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mls-mpm_b200", "csrc")
SOURCE = """
#include "mpm_stencil.h"
extern "C" int in(int32_t c, int32_t lo, int32_t n) { return mpm::stencil_in(c, lo, n); }
extern "C" int32_t cell(int32_t c, int k) { return mpm::stencil_cell(c, k); }
"""
INT_MIN, INT_MAX = -(1 << 31), (1 << 31) - 1


@pytest.mark.parametrize("opt", ["-O0", "-O2", "-O3"])
def test_stencil_tests_hold_for_every_cell(tmp_path, opt):
    src, lib = tmp_path / "s.cpp", tmp_path / "s.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", opt, "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)],
                   check=True)
    f = ctypes.CDLL(str(lib))
    for lo in (-1, 0, 1, 15, 1023):                       # a grid from 0, a chunk's box from one cell before a tile
        for n in (3, 5, 18, 24, 128, 1 << 20, (1 << 29) - 1):
            near = [lo + d for d in range(-3, 4)] + [lo + n + d for d in range(-4, 4)] + [lo + n // 2]
            for c in near + [0, -1, INT_MIN, INT_MIN + 1, INT_MIN + 2, INT_MAX, INT_MAX - 1, INT_MAX - 2, 1 << 30, -(1 << 30)]:
                assert bool(f["in"](c, lo, n)) == (lo <= c - 1 and c + 1 < lo + n), (c, lo, n)
    for c in (INT_MIN, INT_MIN + 1, -1, 0, 1, 127, INT_MAX - 1, INT_MAX):
        for k in range(3):
            want = (c - 1 + k + (1 << 31)) % (1 << 32) - (1 << 31)
            assert f["cell"](c, k) == want
            # no wrapped cell lies in a grid
            assert (0 <= want < 1 << 29) == (0 <= c - 1 + k < 1 << 29)
