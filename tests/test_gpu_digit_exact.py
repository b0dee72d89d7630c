"""Digit products whose digits are in step with the matrix's: the sums of a level pass 2^24, where FP32 no longer
holds every integer, at lengths from about 450 on (and from about 300 on where the matrix holds a factor).

Inputs are made of four digits (of 9 bits) each, which the sign of the matrix's digits is given to, so that
every product of level 3 of one output has the same sign.  A unit of level 3 is 2^-41 of the largest input.
Tolerance, for inputs up to 1: results rounded to FP64 twice, and 550 inputs held to 2^-58 (below 2^-47)."""
import numpy as np
import pytest

from specter_gb300 import api

pytestmark = pytest.mark.gpu
LD = np.longdouble


def close(got, want):
    return np.all(np.abs(got.astype(LD) - want) < np.abs(want) * 2.0**-52 + 2.0**-47)


def plan(nx, ny, nz, Lz=1.0):
    return api.Plan((nx, ny, nz), (0, 0, 25), (0, 0, 5), (1.0, 1.0, Lz), precision=api.FP64)


def angle(a, n):
    pi = LD(np.pi) + LD(1.2246467991473532e-16)
    return 2 * pi * (a % n).astype(LD) / n


def against(t, top=255):
    """A number (in units of 2^-60) whose digit i has the sign of digit 3 - i of t, |t| <= 1."""
    v = np.rint(np.asarray(t, np.float64) * 2.0**53).astype(np.int64) << 9  # 2^62 is 1
    d, rest = [], v
    for i in range(4):  # signed digits: nearest multiples from the top
        u = 54 - 9 * i
        q = (rest + (1 << (u - 1))) >> u if i else (rest + sum(256 << (54 - 9 * j) for j in range(1, 7))) >> 54
        d.append(q)
        rest = rest - (q << u)
    s = [np.where(x < 0, -1, 1) for x in d]
    return sum((top if i == 0 else 255) * s[3 - i].astype(np.int64) << (54 - 9 * i) for i in range(4))


@pytest.mark.parametrize("n", [450, 512, 538, 550])
def test_columns(n):
    p = plan(16, 6, n)
    m = n // 2
    k = np.arange(1, (m + 1) // 2)  # k, m - k, m + k, n - k are four
    js = np.arange(p.nxh * 6) * 2 + 2  # even frequencies
    a, want = np.zeros((len(js), n)), np.zeros(len(js), LD)
    for c, f in enumerate(js):
        cos = np.cos(angle(f * k, n))
        v = against(cos)
        x = v * 2.0**-62
        assert np.all(x * 2.0**62 == v)
        for q in (k, m - k, m + k, n - k):
            a[c, q] = x
        want[c] = np.sum(4 * x.astype(LD) * cos)
    f = p.field(data=(a + 0j).reshape(p.sshape))
    api.fftp1d_complex_to_real_z(p, f)
    got = f.download().reshape(len(js), n)[np.arange(len(js)), js % n]
    assert close(got.real, want)


# The y pass beside the x pass sees one row in ny only, and so keeps every value.
@pytest.mark.parametrize("n", [450, 512, 550])
def test_rows(n):
    nz = 58
    p = plan(n, 2, nz)
    m = n // 2
    # real rows: the sine list of an even frequency
    k = np.arange(1, (m + 1) // 2)
    fs = np.arange(nz) * 2 + 2
    r, want = np.zeros(p.rshape), np.zeros(nz, LD)
    for c, f in enumerate(fs):
        sin = np.sin(angle(f * k, n))
        x = against(sin) * 2.0**-62
        for q, s in ((k, 1), (m + k, 1), (m - k, -1), (n - k, -1)):
            r[c, 0, q] = s * x
        want[c] = -np.sum(4 * x.astype(LD) * sin)
    i, o = p.field(api.REAL, data=r), p.field()
    api.fftp2d_real_to_complex_xy(p, i, o)
    got = o.download()[fs, 0, np.arange(nz)]
    assert close(got.imag, want)
    # half spectra: the cosines of the even frequencies at one point
    k = np.arange(1, (m - 1) // 2 + 1)
    pts = np.arange(nz) + 1
    h, want = np.zeros(p.sshape, complex), np.zeros(nz, LD)
    for c, j in enumerate(pts):
        cos = np.cos(angle(2 * k * j, n))
        x = against(cos, 127) * 2.0**-61
        h[2 * k, 0, c] = x
        want[c] = np.sum(2 * x.astype(LD) * cos)
    o.upload(h)
    api.fftp2d_complex_to_real_xy(p, o, i)
    got = i.download()[np.arange(nz), 0, pts]
    assert close(got, want)
