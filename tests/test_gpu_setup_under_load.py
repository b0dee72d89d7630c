"""A plan's tables are there before its first kernel, however busy the device is: solvers set up while others run give
the same bits as on an idle device."""
import threading
import time

import numpy as np
import pytest

from specter_gb300 import api

pytestmark = pytest.mark.gpu


def solver(nx, ny, nzp, kind=api.BOUSS):
    p = api.Plan((nx, ny, nzp + 25), (0, 0, 25), (0, 0, 5), (1.0, 1.0, 1.0), precision=api.FP32)
    return p, api.Solver(p, kind, ord=2, dt=1e-5, nu=1e-4, kappa=1e-4)


def run(nx, ny, nzp):
    p, s = solver(nx, ny, nzp)
    rng = np.random.default_rng(nzp)
    r = p.field(api.REAL, data=(1e-3 * rng.standard_normal(p.rshape)).astype(np.float32))
    api.fftp3d_real_to_complex(p, r, s.th)
    s.step(3)
    out = [f.download() for f in s.state]
    s.close()
    return out


def leave_nan():
    """Freed memory of the sizes that tables have, holding NaN."""
    fields = []
    for nx, ny, nz, count in ((8, 2, 36, 60), (8, 4, 58, 60), (16, 8, 90, 30), (32, 16, 90, 10)):
        p = api.Plan((nx, ny, nz), (0, 0, 25), (0, 0, 5), (1.0, 1.0, 1.0), precision=api.FP64)
        nan = np.full(p.sshape, np.nan + 1j * np.nan)
        fields += [p.field(data=nan) for _ in range(count)]
    for f in fields:
        f.close()


def test_setup_under_load():
    grids = [(64, 64, 257), (64, 128, 257)]
    want = {g: run(*g) for g in grids}
    busy = [solver(*g) for g in ((256, 128, 257), (128, 256, 257), (128, 128, 257), (256, 256, 129), (64, 256, 257),
                                 (256, 256, 257), (128, 64, 129), (256, 64, 65), (64, 64, 129))]
    graphs = [api.Graph([s]) for _, s in busy]
    stop = threading.Event()

    def drive():  # as the server does
        while not stop.is_set():
            for q in graphs:
                if q.done():
                    for _ in range(25):
                        q.launch()
            time.sleep(2e-4)

    t = threading.Thread(target=drive)
    t.start()
    try:
        differs = []
        for g in grids:
            leave_nan()
            if not all(np.array_equal(a, b) for a, b in zip(run(*g), want[g])):
                differs.append(g)
    finally:
        stop.set()
        t.join()
    for q in graphs:
        q.synchronize()
    assert not differs
