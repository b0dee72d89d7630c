"""FP64 plans with digit-product transforms beside one another and at the limits of their workspace."""
import threading

import numpy as np
import pytest

from specter_gb300 import api

pytestmark = pytest.mark.gpu


def plan(nx, ny, nz, precision=api.FP64):
    return api.Plan((nx, ny, nz), (0, 0, 25), (0, 0, 5), (1.0, 1.0, 1.0), precision=precision)


# Plans of different lengths on threads of their own: they run the same kernels with other shared memory.
@pytest.mark.parametrize("precision", [api.FP64, api.FP32], ids=["fp64", "fp32"])
def test_threads(precision):
    lens = (58, 300, 154, 538, 90, 282)
    start, errors = threading.Barrier(len(lens)), []

    def work(nz):
        try:
            p = plan(4, 2, nz, precision)
            f = p.field()
            start.wait()
            for i in range(4000):
                api.fftp1d_complex_to_real_z(p, f)
                if i % 200 == 0:
                    p.synchronize()
            p.synchronize()
        except Exception as e:
            errors.append((nz, e))
            start.abort()

    ts = [threading.Thread(target=work, args=(n,)) for n in lens]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors


# A transform kernel that gave up a wait leaves wrong results: whatever waits for them or hands them out fails.
def test_gave_up_is_reported():
    p = plan(32, 32, 58)
    s = api.Solver(p, api.HD, ord=2, dt=1e-4, nu=1e-3)
    g = api.Graph([s])
    r, f = p.field(api.REAL), p.field()
    host = [np.empty(f.shape, f.dtype) for _ in range(2)]
    calls = {
        "transform": lambda: api.fftp1d_complex_to_real_z(p, f),
        "rows": lambda: api.fftp2d_real_to_complex_xy(p, r, f),
        "step": lambda: s.step(1),
        "synchronize": p.synchronize,
        "download": f.download,
        "fields": lambda: api.fields_download([f, s.vx], [a.ctypes.data for a in host]),
        "energy": lambda: api.energy(p, f, f, f, 1),
        "walls": lambda: api.bouncheck_z(p, f, f),
        "static walls": lambda: api.bouncheck_z_static(p, f, f),
        "check": s.check,
        "replay": g.launch,
        "replayed": g.synchronize,
        "replay done": g.done,
    }
    for c in calls.values():
        c()
    p.synchronize()
    api.set_option(p, "gave_up", 1)  # as the kernel does, from the host
    ok = []
    for name, c in calls.items():
        try:
            c()
            ok.append(name)
        except api.SpecterError as e:
            assert e.code == 5 and "gave up" in str(e)
    assert not ok
    api.set_option(p, "gave_up", 0)
    for c in calls.values():
        c()
