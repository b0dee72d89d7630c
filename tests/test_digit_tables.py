"""The digit matrices and what their sums can be trusted with (csrc/tctables.h, compiled for the host)."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "specter_gb300", "csrc")
SRC = """
#include "tctables.h"
extern "C" int digits(int n, double factor, int half, int *c, int *s, int *expo, double *post, float *top, int *nq) {
    const sg::Dims D = sg::dims(n);
    sg::MatrixDigits m;
    if (!sg::matrix_digits_for(D, factor, half, m)) return 1;
    for (int t = 0; t < n; t++)
        for (int i = 0; i < sg::kDig; i++) {
            c[t * sg::kDig + i] = m.digit(n, false, t, i);
            s[t * sg::kDig + i] = m.digit(n, true, t, i);
        }
    *expo = m.expo;
    *post = m.post;
    top[0] = m.top[0];
    top[1] = m.top[1];
    nq[0] = D.nq[0];
    nq[1] = D.nq[1];
    return 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tables")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "t.so"), str(d / "t.cpp")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("n", [32, 34, 58, 154, 282, 320, 400, 450, 512, 538, 550])
@pytest.mark.parametrize("factor", [1.0, "1/n", "dkz", 0.9990234375, 0.7071])
def test_matrix(lib, n, half, factor):
    factor = {"1/n": 1 / n, "dkz": 2 * math.pi * (n - 26) / n}.get(factor, factor)
    c, s = np.zeros((n, 7), np.int32), np.zeros((n, 7), np.int32)
    expo, post, top, nq = ctypes.c_int(), ctypes.c_double(), (ctypes.c_float * 2)(), (ctypes.c_int * 2)()
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (c, s)]
    assert lib.digits(n, ctypes.c_double(factor), half, p[0], p[1], ctypes.byref(expo), ctypes.byref(post), top, nq) == 0
    # the digits are the numbers: digit 0 in units of 2^-8 of one
    w = 2.0 ** (-8 - 9 * np.arange(7))
    t = 2 * np.pi * np.arange(n) / n
    got = math.ldexp(post.value, expo.value) * np.stack([c @ w, s @ w])
    assert np.max(np.abs(got - factor * np.stack([np.cos(t), np.sin(t)]))) < 4e-15 * factor * max(1, n / 100)
    assert max(np.abs(c).max(), np.abs(s).max()) <= 256
    # the largest sum of a level that data digits up to 256 can make, in any order of its terms
    K, bound = n // 4 + 1, np.zeros(5)
    for d in (c, s):
        a = np.abs(d)
        for par in range(2):
            pts, fqs = np.arange(K), np.arange(nq[par])
            ang = (2 * fqs[:, None] + par) * pts[None, :] % n
            if half:
                ang = ang.T
            for v in range(5):
                bound[v] = max(bound[v], 256 * a[ang][..., : v + 1].sum(axis=(1, 2)).max())
    assert max(bound[:3]) <= 2**24
    for v in (0, 1):  # a partial sum beyond 2^24 cannot end below top
        assert top[v] >= 2**22
        assert math.isinf(top[v]) and bound[3 + v] <= 2**24 or 2**24 - (bound[3 + v] - 2**24) >= top[v]
