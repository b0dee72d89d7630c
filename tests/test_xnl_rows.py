"""Rows a block of the FP32 nonlinear x pass (csrc/xnlrows.h, compiled for the host)."""
import ctypes
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "specter_gb300", "csrc")


def test_rows(tmp_path):
    (tmp_path / "r.cpp").write_text('#include "xnlrows.h"\n'
                                    'extern "C" int rows(int rb, int pipelined, int pair, int asked) { return sg::xnl_rows(rb, pipelined, pair, asked); }\n')
    lib = str(tmp_path / "r.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", lib, str(tmp_path / "r.cpp")], check=True)
    rows = ctypes.CDLL(lib).rows
    assert rows(16, 1, 0, 0) == 8  # nx = 512 with no cap of its own
    assert rows(16, 1, 0, 1) == 16  # and with a cap of 16
    for rb in (1, 2, 4, 8, 16):
        assert rows(rb, 1, 1, 0) == rows(rb, 0, 0, 0) == rows(rb, 0, 0, 1) == rb
        assert rb == 16 or rows(rb, 1, 0, 0) == rows(rb, 1, 0, 1) == rb
