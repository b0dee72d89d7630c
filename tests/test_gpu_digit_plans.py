"""FP64 plans with digit-product transforms beside one another and at the limits of their workspace."""
import threading

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
