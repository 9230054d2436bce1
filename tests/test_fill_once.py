"""fill_once.h, compiled for the host: tables that all contexts of a device share are written by the first
context only (a later one would write while kernels of others read them), also when contexts are created
at the same time, again after a fill that failed, and again on a device that has lost them."""
import ctypes as C
import os
import subprocess

from conftest import ROOT

SHIM = """
#include <atomic>
#include <thread>
#include <vector>
#include "fill_once.h"
namespace {
std::atomic<int> fills{0}, inside{0}, overlaps{0}, marked{0};
int init(int fail) {
  return cz::fill_once([](bool* done) { *done = marked != 0; return 0; },
                       [&] {
                         if (inside++) overlaps++;
                         std::this_thread::yield();
                         fills++;
                         inside--;
                         return fail;
                       },
                       [] { marked = 1; return 0; });
}
}
extern "C" int init_from(int threads, int fail) {
  std::vector<std::thread> t;
  std::atomic<int> rc{0};
  for (int i = 0; i < threads; i++) t.emplace_back([&] { rc |= init(fail); });
  for (auto& x : t) x.join();
  return rc;
}
extern "C" int count() { return fills; }
extern "C" int overlapped() { return overlaps; }
extern "C" void lose() { marked = 0; }
"""


def test_shared_tables_are_filled_once(tmp_path):
    (tmp_path / "shim.cpp").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread",
                           "-I" + os.path.join(ROOT, "collatz_b200", "csrc"), str(tmp_path / "shim.cpp"), "-o", so])
    L = C.CDLL(so)
    assert L.init_from(1, 7) == 7 and L.count() == 1  # a fill that failed does not count
    assert L.init_from(16, 0) == 0 and L.count() == 2 and L.overlapped() == 0
    assert L.init_from(16, 0) == 0 and L.count() == 2
    L.lose()
    assert L.init_from(4, 0) == 0 and L.count() == 3


def test_the_kernels_tables_are_filled_through_it():
    """The table kernels are launched from inside fill_once and nowhere else."""
    for name, kernel in (("range.cu", "k_win_tables<<<"), ("cases_win.cu", "k_cp_tables<<<")):
        with open(os.path.join(ROOT, "collatz_b200", "csrc", name)) as f:
            src = f.read()
        assert src.count(kernel) == 1
        assert src[:src.index(kernel)].rindex("fill_once(") > src[:src.index(kernel)].rindex("\ncudaError_t ")
