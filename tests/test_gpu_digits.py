"""FP64 column transforms as digit products on the tensor cores, against numpy's FP64 FFT, at the edges
of their range: the shortest and longest lengths, halves that are odd, tiles of columns that end
inside a column tile, columns of very different size, zero and non-finite columns.

Tolerance: a double-precision FFT of up to 550 points is within 1e-15 of the exact transform (relative
L2 of a column), the digit products within 3e-16: 2e-15 between the two."""
import numpy as np
import pytest

from conftest import make_pair, rel, smooth_spectral
from specter_gb300 import api

pytestmark = pytest.mark.gpu
TOL = 2e-15


def plan(nx, ny, nz):
    return api.Plan((nx, ny, nz), (0, 0, 25), (0, 0, 5), (1.0, 1.0, 1.0), precision=api.FP64)


def col_err(a, b):
    m = np.abs(b).max(axis=-1, keepdims=True)
    return np.max(np.linalg.norm((a - b) / m, axis=-1) / np.linalg.norm(b / m, axis=-1))


@pytest.mark.parametrize("nz", [36, 38, 58, 62, 64, 90, 154, 158, 160, 282, 318, 320, 322, 512, 538, 550, 552])
@pytest.mark.parametrize("nx,ny", [(8, 4), (36, 6)])
def test_z_inverse(nx, ny, nz):
    p = plan(nx, ny, nz)
    rng = np.random.default_rng(nz)
    a = rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)
    a[0] *= np.exp(-np.minimum(np.arange(nz), nz - np.arange(nz)))  # a few large modes
    a[1, 0] *= 1e-290
    a[1, 1] *= 1e290
    a[1, 2] = 0
    a[1, 2, nz // 2] = 1.0
    a[2, 0] = 0
    f = p.field(data=a)
    api.fftp1d_complex_to_real_z(p, f)
    got, want = f.download(), np.fft.ifft(a, axis=-1) * nz
    assert np.all(got[2, 0] == 0)
    got[2, 0] = want[2, 0] = 1
    assert col_err(got, want) < TOL


@pytest.mark.parametrize("ny", [30, 32, 34, 62, 66, 100, 256, 512])
def test_xy_round_trip(ny):
    p = plan(16, ny, 36)
    rng = np.random.default_rng(ny)
    r = rng.standard_normal(p.rshape)
    f, c, o = p.field(api.REAL, data=r), p.field(), p.field(api.REAL)
    api.fftp2d_real_to_complex_xy(p, f, c)
    want = np.fft.rfft2(r).transpose(2, 1, 0)
    got = c.download()
    assert np.linalg.norm(got - want) < TOL * np.linalg.norm(want)
    api.fftp2d_complex_to_real_xy(p, c, o)
    assert np.linalg.norm(o.download() / (16 * ny) - r) < TOL * np.linalg.norm(r)


@pytest.mark.parametrize("nx", [94, 96, 98, 130, 254, 256, 512, 550])
def test_x_rows(nx):
    p = plan(nx, 6, 36)  # 216 rows: the second tile of 128 is not full
    rng = np.random.default_rng(nx)
    r = rng.standard_normal(p.rshape)
    r[3, 2] *= 1e-200
    r[4, 1] = 0
    f, c, o = p.field(api.REAL, data=r), p.field(), p.field(api.REAL)
    api.fftp2d_real_to_complex_xy(p, f, c)
    want = np.fft.rfft2(r).transpose(2, 1, 0)
    assert np.linalg.norm(c.download() - want) < TOL * np.linalg.norm(want)
    # any half spectrum: the imaginary parts of frequencies 0 and nx/2 do not count (of the y transform's
    # results, as of irfft's input)
    a = rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)
    c.upload(a)
    api.fftp2d_complex_to_real_xy(p, c, o)
    y = np.fft.ifft(a.transpose(2, 1, 0), axis=1) * 6
    want = np.fft.irfft(y, n=nx, axis=2) * nx
    assert np.linalg.norm(o.download() - want) < TOL * np.linalg.norm(want)


# short rows, on both sides of the number of rows from which they are digit products (2048)
@pytest.mark.parametrize("nx", [32, 34, 64, 94])
@pytest.mark.parametrize("ny", [56, 58])
def test_short_x_rows(nx, ny):
    p = plan(nx, ny, 36)
    rng = np.random.default_rng(nx + ny)
    r = rng.standard_normal(p.rshape)
    f, c, o = p.field(api.REAL, data=r), p.field(), p.field(api.REAL)
    api.fftp2d_real_to_complex_xy(p, f, c)
    want = np.fft.rfft2(r).transpose(2, 1, 0)
    assert np.linalg.norm(c.download() - want) < TOL * np.linalg.norm(want)
    a = rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)
    c.upload(a)
    api.fftp2d_complex_to_real_xy(p, c, o)
    y = np.fft.ifft(a.transpose(2, 1, 0), axis=1) * ny
    want = np.fft.irfft(y, n=nx, axis=2) * nx
    assert np.linalg.norm(o.download() - want) < TOL * np.linalg.norm(want)


def test_non_finite_and_denormal_columns():
    p = plan(8, 4, 58)
    rng = np.random.default_rng(0)
    a = rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)
    a[1, 1, 7] = np.inf
    a[2, 2, 5] = np.nan
    a[3, 3] *= 1e-310
    a[0, 1] *= 1e307
    f = p.field(data=a)
    api.fftp1d_complex_to_real_z(p, f)
    got = f.download()
    assert np.all(np.isnan(got[1, 1].real)) and np.all(np.isnan(got[2, 2].real))
    with np.errstate(invalid="ignore", over="ignore"):
        want = np.fft.ifft(a, axis=-1) * 58
    # denormal results are rounded to multiples of 2^-1074
    assert np.max(np.abs(got[3, 3] - np.fft.ifft(a[3, 3] * 2.0**60) * 58 * 2.0**-60)) <= 2.0**-1073
    ok = np.ones(p.sshape[:2], bool)
    ok[1, 1] = ok[2, 2] = ok[3, 3] = ok[0, 1] = False
    assert col_err(got[ok], want[ok]) < TOL
    big = np.fft.ifft(a[0, 1] * 2.0**-60) * 58
    fits = (np.abs(big.real) < 1e289) & (np.abs(big.imag) < 1e289)
    assert np.allclose(got[0, 1][fits] * 2.0**-60, big[fits], rtol=1e-12, atol=0)


# the x pass of the nonlinear term and the whole plain FP64 stage: shortest and longest lengths, halves
# that are odd, rows that end inside a tile of 128.  1e-11: the continuation amplifies rounding by 1e4
# (tests/test_gpu_parity.py).
@pytest.mark.parametrize("nx,ny,nzp", [(32, 4, 33), (34, 6, 29), (62, 10, 11), (100, 32, 13), (254, 4, 11), (512, 4, 11),
                                       (550, 2, 11)])
def test_nonlinear_term(nx, ny, nzp):
    p, g = make_pair(nx, ny, nzp, 1.0)
    rng = np.random.default_rng(nx)
    v = [smooth_spectral(g, rng) for _ in range(4)]
    f, out = [p.field(data=a) for a in v], [p.field() for _ in range(4)]
    api.gradre(p, f[0], f[1], f[2], out[0], out[1], out[2])
    api.advect(p, f[0], f[1], f[2], f[3], out[3])
    want = list(g.gradre(*v[:3])) + [g.advect(*v[:3], v[3])]
    for a, b in zip(out, want):
        assert rel(a.download(), b) < 1e-11
