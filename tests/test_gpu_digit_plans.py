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


def room(p, mb):
    api.set_option(p, "digit_room_mb", mb)
    return p


# Room for a few tiles of digits: the same launches in ranges of tiles, or one transform at a time, bit for bit.
@pytest.mark.parametrize("nx,ny,nz", [(96, 40, 58), (34, 64, 90), (130, 34, 154)])
def test_ranges(nx, ny, nz):
    def run(p):
        rng = np.random.default_rng(nx)
        r = p.field(api.REAL, data=rng.standard_normal(p.rshape))
        f = [p.field(data=rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)) for _ in range(4)]
        o = [p.field() for _ in range(5)]
        out = []
        api.fftp3d_real_to_complex(p, r, o[4])
        api.gradre(p, f[0], f[1], f[2], o[0], o[1], o[2])
        api.advect(p, f[0], f[1], f[2], f[3], o[3])
        out += [x.download() for x in o]
        api.fftp3d_complex_to_real(p, o[4], r)
        o[4].zero()
        api.v_imposebc_and_project(p, f[0], f[1], f[2], o[4], 1, 2)
        return out + [x.download() for x in f + [o[4]]] + [r.download()]

    got, want = run(room(plan(nx, ny, nz), 2)), run(plan(nx, ny, nz))
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("kind", [api.HD, api.BOUSS, api.ROTBOUSS])
def test_stage_ranges(kind):
    def run(mb):
        p = room(plan(96, 40, 90), mb)
        s = api.Solver(p, kind, ord=2, dt=1e-4, nu=1e-3, kappa=1e-3, omega=(0.1, 0.0, 0.5))
        rng = np.random.default_rng(1)
        for f in s.state[:-1]:
            r = p.field(api.REAL, data=1e-2 * rng.standard_normal(p.rshape))
            api.fftp3d_real_to_complex(p, r, f)
        s.step(2)
        return [f.download() for f in s.state]

    small, large, general = run(2), run(0), run(-1)
    assert all(np.array_equal(a, b) for a, b in zip(small, large))
    # against the column kernels on the general engine: rounding times 1e4 (the continuation)
    assert all(np.linalg.norm(a - b) < 1e-11 * np.linalg.norm(b) for a, b in zip(small, general))


# A plan that transforms fields one by one holds the digits of one, not those of the nonlinear term.
def test_memory_of_single_transforms():
    p = plan(128, 128, 154)
    r, c = p.field(api.REAL), p.field()
    p.synchronize()
    free = api.device_memory()[0]
    api.fftp3d_complex_to_real(p, c, r)
    p.synchronize()
    assert free - api.device_memory()[0] < 8 * 16 * 72 * 128 * 154


# An FP64 solver in the memory that it took before its transforms had buffers (about 40 fields, 0.9 GB).
def test_little_memory():
    import torch
    shape = (128, 128, 154)

    def run():
        p = plan(*shape)
        s = api.Solver(p, api.BOUSS, ord=2, dt=1e-4, nu=1e-3, kappa=1e-3)
        rng = np.random.default_rng(1)
        for f in s.state[:-1]:
            f.upload(1e-3 * (rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)))
        s.step(2)
        out = [f.download() for f in s.state]
        s.close()
        p.close()
        return out

    want = run()
    torch.cuda.empty_cache()
    held = torch.empty(api.device_memory()[0] - 1300 * 2**20, dtype=torch.uint8, device="cuda")
    try:
        got = run()
    finally:
        del held
        torch.cuda.empty_cache()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


# The first transform of a plan inside a stream capture, where nothing can be allocated, and one after it.
@pytest.mark.parametrize("before", [False, True])
def test_first_call_captured(before):
    import torch
    w = room(plan(16, 4, 58), -1)
    api.fftp1d_complex_to_real_z(w, w.field())  # its kernel is loaded
    p = plan(16, 4, 58)
    rng = np.random.default_rng(2)
    a = rng.standard_normal(p.sshape) + 1j * rng.standard_normal(p.sshape)
    f, src = p.field(data=a), p.field(data=a)
    if before:
        api.fftp1d_complex_to_real_z(p, f)
    p.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(p.stream)):
        f.copy_from(src)
        api.fftp1d_complex_to_real_z(p, f)
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        want = np.fft.ifft(a, axis=-1) * 58
        assert np.linalg.norm(f.download() - want) < 2e-15 * np.linalg.norm(want)


# What the server reserves for an FP64 request before it has seen one of its kind.
def test_server_estimate():
    from specter_gb300 import serve
    srv = serve.Server(1, precision=0)
    for kind, nx, ny, nzp in (("HD", 64, 64, 65), ("BOUSS", 128, 64, 129), ("BOUSS", 128, 128, 65), ("HD", 256, 64, 257)):
        req = serve.Request(0, 0.0, kind, nx, ny, nzp, 1, 1)
        p, s = serve.make(srv.api, srv.initial, req, 0)
        s.step(1)
        p.synchronize()
        assert api.solver_memory(s) <= srv._estimate(req)
        s.close()
        p.close()


# A plan's first transform is queued like the others: its tables wait for nothing that is queued before them.
def test_first_call_does_not_wait():
    import torch
    w, p = plan(64, 64, 90), plan(64, 64, 90)
    for q in (w, p):
        f = q.field()
        q.synchronize()
        e = torch.cuda.Event()
        with torch.cuda.stream(torch.cuda.ExternalStream(q.stream)):
            torch.cuda._sleep(400_000_000)  # 0.2 s
            e.record()
        api.fftp1d_real_to_complex_z(q, f)
        done = e.query()  # of the second plan, whose kernels are loaded
        q.synchronize()
    assert not done
