"""Which body a range launch runs with (range_variants.h, compiled for the host): short launches get 24
warps per block whichever thresholds are set, by choice or by the autotuner; two variants fix the warps."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT

SHIM = """
#include "range_variants.h"
extern "C" int variants() { return cz::RANGE_VARIANTS; }
extern "C" uint32_t warps_of(int v, unsigned long long rows, uint32_t sms) { return cz::range_pick(v, rows, sms).warps; }
extern "C" uint32_t jw_of(int v) { return cz::range_pick(v, 1, 148).jw; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("variants")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "collatz_b200", "csrc"),
                           str(d / "shim.cpp"), "-o", so])
    L = C.CDLL(so)
    L.warps_of.argtypes = [C.c_int, C.c_ulonglong, C.c_uint32]
    return L


def test_warps_by_rows_for_every_thresholds(lib):
    line = 512 * 32 * 148
    fixed = {6: 32, 7: 24}
    for v in range(lib.variants()):
        for rows, want in [(1, 24), (line - 1, 24), (line, 32), (1 << 50, 32)]:
            assert lib.warps_of(v, rows, 148) == fixed.get(v, want), (v, rows)
        assert lib.jw_of(v) in (12, 13)
