"""The limits up to which the table-driven cases kernel runs a seed by look-ups (case_limits.h, compiled here
for the host): they never pass what could change a line's outputs, and lines of small N have one too."""
import ctypes as C
import os
import random
import subprocess

import pytest

from conftest import ROOT

SHIM = """
#include "case_limits.h"
extern "C" uint32_t unit_of(uint32_t n) { return cz::line_unit(n); }
extern "C" uint32_t limits_of(unsigned long long s, unsigned long long e, uint32_t mbi, uint32_t cap, uint32_t unit) {
  return cz::line_limits(s, e, mbi, cap, unit);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("limits")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "collatz_b200", "csrc"),
                           str(d / "shim.cpp"), "-o", so])
    L = C.CDLL(so)
    L.unit_of.restype = L.limits_of.restype = C.c_uint32
    L.limits_of.argtypes = [C.c_ulonglong, C.c_ulonglong, C.c_uint32, C.c_uint32, C.c_uint32]
    return L


def _key(x):
    b = x.bit_length()
    return (b << 54) | (x >> (b - 54) if b > 54 else x << (54 - b)) if x else 0


@pytest.mark.parametrize("n", [16, 26, 30, 34, 35, 36, 40, 44, 45, 48, 52])
def test_value_limit(lib, n):
    unit = lib.unit_of(n)
    rng = random.Random(n)
    for _ in range(2000):
        bits = rng.randrange(1, 126)
        top = rng.getrandbits(bits) | (1 << (bits - 1))
        word = lib.limits_of(500, _key(top), n - 10, 1 << 16, unit)
        limit = (word & 0xFFFFFF) << (32 + unit)
        # a look-up's odd runs raise a value by less than 1.5^12 < 256, and three words hold 2^96
        assert limit * 256 <= top and limit <= 1 << 71
        # the largest value that is seen before a seed leaves the loop fits the word that is compared
        assert limit << 8 <= 1 << (64 + unit)
        if top < 1 << 60 + unit and top >= 1 << 40 + unit:
            assert (limit + (1 << 32 + unit)) * 256 > top  # no coarser than a unit
    if n <= 45:  # the checkpoint loop's largest start lies below the largest limit
        assert 2 ** n * 3 ** (n - 10) * 32 <= 2 ** (55 + unit) * 2 ** (n - 10)


def test_small_lines_have_a_limit(lib):
    """The maxima of lines of a few thousand seeds: with units of 2^48 for every N these had none, and
    all their seeds ran exactly."""
    for n, bits in [(26, 42), (30, 46), (36, 50), (40, 54)]:
        assert lib.limits_of(200, _key(1 << bits), n - 10, 1 << 16, lib.unit_of(n)) & 0xFFFFFF > 0


@pytest.mark.parametrize("cap", [0, 1, 2, 200, 201, 1 << 16])
def test_look_up_limit(lib, cap):
    for st in (0, 1, 26, 27, 38, 39, 40, 400, 5000, 1 << 25):
        word = lib.limits_of(st, _key(1 << 70), 26, cap, 16)
        k = word >> 24
        if word == 0:  # every seed runs exactly
            assert cap == 0 or st < 26 + 12 or cap == 1
            continue
        assert k <= min(cap, 201) - 1
        assert k == 0 or 26 + 12 * k < st
