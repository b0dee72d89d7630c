"""The state of the precision form: pairs of floats, each the nearest to what is left of the double, down to values
whose second float is a denormal one."""
import numpy as np
import pytest

from specter_gb300 import api

pytestmark = pytest.mark.gpu


def test_pairs_of_small_values():
    plan = api.Plan((64, 16, 58), (0, 0, 25), (0, 0, 5), (1.0, 1.0, 2.0), precision=api.FP64)
    s = api.Solver(plan, api.BOUSS, fused=True, nl_fp32=True, dt=1e-5, nu=1e-4, kappa=1e-4)
    rng = np.random.default_rng(7)
    fields = (s.vx, s.vy, s.vz, s.th, s.pr)
    data = []
    for f in fields:
        a = np.empty(plan.sshape, complex)
        for part in (a.real, a.imag):
            part[...] = (1 + rng.random(plan.sshape)) * 2.0 ** rng.integers(-130, -80, plan.sshape) * rng.choice([-1, 1], plan.sshape)
        data.append(a)
        f.upload(a)
    s.step(0)  # to pairs and back
    for f, a in zip(fields, data):
        b = f.download()
        for x, y in ((a.real, b.real), (a.imag, b.imag)):
            hi = x.astype(np.float32)
            lo = (x - hi).astype(np.float32)
            assert np.array_equal(y, hi.astype(float) + lo.astype(float))
