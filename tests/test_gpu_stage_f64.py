"""The plain FP64 stage over the digit transforms (csrc/stage_f64.cu) at the edges of their lengths, against the oracle:
the shortest z lengths (halves even and odd), the longest, and one past it, where the column kernels run.

Tolerance: the continuation's row sums (9.5e3) times FP64 rounding, about twenty times in two steps: 5e-11."""
import numpy as np
import pytest

from conftest import make_pair, rel, smooth_spectral
from specter_gb300 import api

pytestmark = pytest.mark.gpu
OMEGA = (0.1, 0.0, 0.5)


@pytest.mark.parametrize("kind", [api.HD, api.BOUSS, api.ROTBOUSS])
@pytest.mark.parametrize("nx,ny,nzp", [(32, 32, 11), (34, 34, 13), (32, 6, 39), (36, 4, 525), (32, 6, 527)])
def test_stage_at_edges(kind, nx, ny, nzp):
    plan, g = make_pair(nx, ny, nzp, 1.0)
    rng = np.random.default_rng(nzp + kind)
    v = [smooth_spectral(g, rng, amp=0.3) for _ in range(3)]
    th = smooth_spectral(g, rng, amp=0.3)
    pr = np.zeros(g.sshape, complex)
    kw = dict(dt=1e-4, nu=1e-3, ord=2, kappa=5e-4)
    s = api.Solver(plan, kind, fused=True, omega=OMEGA if kind == api.ROTBOUSS else (0.0, 0.0, 0.0), **kw)
    for f, a in zip((s.vx, s.vy, s.vz, s.pr), v + [pr]):
        f.upload(a)
    if kind != api.HD:
        s.th.upload(th)
    s.step(2)
    ref = g.run(g.params(**kw), 2, *v, pr, th=th if kind != api.HD else None, omega=OMEGA if kind == api.ROTBOUSS else None)
    got = [f.download() for f in s.state[:-1]]
    for a, b in zip(got, ref):
        assert rel(a, b) < 5e-11
