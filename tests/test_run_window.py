"""Window plans of the run-layout solves (csrc/run_window.h), on the host: a
window is said to fit only when its elements do, however large the image."""
import ctypes as ct
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "geopyv-dev_b200", "csrc")
SRC = """
#include "run_window.h"
extern "C" int plan(int banks, int xlo, int xhi, int ylo, int yhi, int border, int cap, int *o) {
    return banks == 16 ? gpv::run_plan<16>(xlo, xhi, ylo, yhi, border, cap, o[0], o[1], o[2], o[3], o[4])
                       : gpv::run_plan<32>(xlo, xhi, ylo, yhi, border, cap, o[0], o[1], o[2], o[3], o[4]);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SRC)
    so = str(d / "plan.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    str(d / "plan.cpp")], check=True)
    f = ct.CDLL(so).plan

    def call(banks, xlo, xhi, ylo, yhi, cap, border=20):
        o = (ct.c_int * 5)()
        return bool(f(banks, xlo, xhi, ylo, yhi, border, cap, o)), list(o)  # r0, c0, wh, ww, pitch
    return call


@pytest.mark.parametrize("banks", [16, 32])
@pytest.mark.parametrize("w,h", [(46400, 46400), (65536, 65536), (92700, 23200), (1 << 30, 2), (65536, 1 << 17)])
def test_whole_large_images_do_not_fit(plan, banks, w, h):
    ok, _ = plan(banks, 0, w - 1, 0, h - 1, 58000)  # 227 KB of floats
    assert not ok


@pytest.mark.parametrize("banks", [16, 32])
@pytest.mark.parametrize("n", [1, 8, 61, 121])
def test_a_window_that_fits_covers_the_taps(plan, banks, n):
    need = (n + 40) * (n + 44)
    ok, (r0, c0, wh, ww, pitch) = plan(banks, 100, 100 + n - 1, 200, 200 + n - 1, need)
    assert ok and pitch * wh <= need and pitch >= ww and pitch % banks and c0 % 4 == 0 and ww % 4 == 0
    assert c0 <= 100 + 20 - 2 and c0 + ww > 100 + n - 1 + 20 + 3
    assert r0 <= 200 + 20 - 2 and r0 + wh > 200 + n - 1 + 20 + 3
    assert not plan(banks, 100, 100 + n - 1, 200, 200 + n - 1, n * n)[0]
