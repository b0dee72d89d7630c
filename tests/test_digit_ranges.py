"""Launches of the digit transforms stay within the digit workspace (csrc/tcranges.h, compiled for the host)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "specter_gb300", "csrc")
SRC = """
#include "tcranges.h"
extern "C" void range(int njobs, unsigned tiles, unsigned long long cap, int *jobs, unsigned *t) {
    const sg::TcRange r = sg::tc_range(njobs, tiles, cap);
    *jobs = r.jobs;
    *t = r.tiles;
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("ranges")
    src, lib = d / "range.cpp", d / "range.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(lib), str(src)], check=True)
    f = ctypes.CDLL(str(lib)).range

    def call(njobs, tiles, cap):
        j, t = ctypes.c_int(), ctypes.c_uint()
        f(njobs, ctypes.c_uint(tiles), ctypes.c_ulonglong(cap), ctypes.byref(j), ctypes.byref(t))
        return j.value, t.value

    return call


# 2112 tiles against 2080: the z columns of 512 x 512 x 538 in a workspace of 2 GiB
@pytest.mark.parametrize("cap", [1, 2, 15, 16, 17, 100, 2080, 2112, 4224])
@pytest.mark.parametrize("tiles", [1, 2, 16, 17, 99, 100, 101, 2080, 2081, 2112, 8712])
@pytest.mark.parametrize("njobs", [1, 2, 3, 8, 15, 16])
def test_every_launch_fits(cut, njobs, tiles, cap):
    jobs, step = cut(njobs, tiles, cap)
    assert 1 <= jobs <= njobs and 1 <= step <= tiles
    assert jobs * step <= cap
    assert jobs == 1 or step == tiles  # several transforms in a launch: whole ones
