"""The one-disk driver (fb_host.c) on a CUDA runtime of the host
(fake_cuda.c), whose streams run as late as the real ones may: what a step
queues reads what that step wrote."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture()
def host(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    so = str(tmp_path / "libhost.so")   # a library of its own per test (its counters start at zero) that keeps to its own runtime
    subprocess.run(["gcc", "-O1", "-std=gnu99", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-ffp-contract=off", "-Dsched_yield=fake_yield",
                    "-I" + os.path.join(CUDA, "include"), "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "fargo3d_b200", "csrc"),
                    os.path.join(ROOT, "fargo3d_b200", "csrc", "fb_host.c"), os.path.join(ROOT, "tests", "fake_cuda.c"),
                    "-o", so, "-lm", "-lpthread"], check=True)
    L = C.CDLL(so)
    L.fb_disk_stream.restype = C.c_void_p
    L.fb_last_error.restype = C.c_char_p
    L.fake_count.argtypes = [C.c_void_p]
    return L


class _Disk:
    def __init__(self, L, **kw):
        from fargo3d_b200 import _abi, config_fargo2d
        self.L, self.h = L, C.c_void_p()
        self.p = _abi.params_of(config_fargo2d(16, 8).replace(**kw))
        self.check(L.fb_disk_create(C.byref(self.p), _abi.FB_FP64, 0, C.byref(self.h)))
        self.stream = C.c_void_p(L.fb_disk_stream(self.h))

    def check(self, rc):
        assert rc == 0, self.L.fb_last_error()

    def begin(self):
        m = C.c_double()
        self.check(self.L.fb_disk_step_begin(self.h, C.byref(m)))
        return m.value

    def advance(self, cfl):
        dt = C.c_double()
        self.check(self.L.fb_disk_step_advance(self.h, C.c_double(1e30), C.c_double(cfl), C.byref(dt)))
        return dt.value

    def transport(self):
        self.check(self.L.fb_disk_step_transport(self.h))

    def step(self):
        dt = C.c_double()
        self.check(self.L.fb_disk_step(self.h, C.c_double(1e30), C.byref(dt)))
        return dt.value

    def sync(self):
        assert self.L.cudaStreamSynchronize(self.stream) == 0

    def close(self):
        self.check(self.L.fb_disk_destroy(self.h))


def _found(L):
    return list((C.c_double * 256).in_dll(L, "fake_dts"))[:C.c_int.in_dll(L, "fake_ndts").value]


@pytest.mark.parametrize("before", [0, 5])   # as launches, as graphs
def test_each_step_reads_its_own_scalars(host, before):
    """A whole step, then advances with the caller's own CFL minimum and no
    begin between: the scalars of a step in flight stay until it has read
    them."""
    d = _Disk(host)
    want = []
    for _ in range(before):
        want.append(d.step())
        want.append(d.advance(0.5 * d.begin()))
        d.transport()
    want.append(d.step())
    for k in range(3):
        want.append(d.advance(0.01 * (k + 1)))
        d.transport()
    d.sync()
    assert _found(host) == want
    d.close()


def test_work_queued_by_others_during_a_capture(host):
    """A part is captured on a stream of its own: what another thread queues
    on the disk's stream meanwhile (a batch's members share one) runs once."""
    d = _Disk(host)
    calls = []

    @C.CFUNCTYPE(None)
    def other():
        calls.append(host.fake_count(d.stream))
    C.c_void_p.in_dll(host, "fake_on_capture").value = C.cast(other, C.c_void_p).value
    for _ in range(12):
        d.advance(0.5 * d.begin())
        d.transport()
        d.step()
    d.sync()
    assert len(calls) >= 3   # begin, advance, transport
    assert C.c_int.in_dll(host, "fake_counted").value == len(calls)
    C.c_void_p.in_dll(host, "fake_on_capture").value = None
    d.close()


def test_parts_inside_a_callers_capture(host):
    """A caller that captures the disk's stream gets the launches of advance
    and transport in its graph, before and after they go out as graphs."""
    d = _Disk(host)
    for _ in range(7):
        d.advance(d.begin())
        d.transport()
        d.step()
        d.sync()
        n = C.c_int.in_dll(host, "fake_ndts").value
        g, e = C.c_void_p(), C.c_void_p()
        assert host.cudaStreamBeginCapture(d.stream, 1) == 0
        dt = d.advance(0.25)
        d.transport()
        assert host.cudaStreamEndCapture(d.stream, C.byref(g)) == 0
        assert C.c_int.in_dll(host, "fake_ndts").value == n   # nothing ran yet
        assert host.cudaGraphInstantiate(C.byref(e), g, C.c_ulonglong(0)) == 0
        for _ in range(2):
            assert host.cudaGraphLaunch(e, d.stream) == 0
        d.sync()
        assert _found(host)[n:] == [dt, dt]
        assert host.cudaGraphDestroy(g) == 0 and host.cudaGraphExecDestroy(e) == 0
    d.close()


@pytest.mark.parametrize("flags", [0, 2, 4])   # automatic, yield, blocking
def test_a_long_begin_leaves_the_core_to_others(host, flags):
    """The begin watches for its report a while, then waits as the process
    chose for the device: blocked in the stream's wait, or yielding."""
    C.c_int.in_dll(host, "fake_lazy_cfl").value = 1
    C.c_int.in_dll(host, "fake_flags").value = flags
    d = _Disk(host)
    now = [C.c_int.in_dll(host, "fake_" + n) for n in ("syncs", "queries", "yields")]
    for _ in range(6):
        was = [n.value for n in now]
        assert d.begin() == 0.125
        syncs, queries, yields = (n.value - w for n, w in zip(now, was))
        if flags == 4:
            assert (syncs, queries) == (1, 0)
        else:
            assert syncs == 0 and queries >= 1 and yields >= 100 * queries
    d.close()


def test_tiles_read_back(host):
    """What get_tiles reports can be set again and changes nothing: 0 where the
    launch's work decides the column segment."""
    d = _Disk(host)
    cx, ns = C.c_int(), C.c_int()

    def get():
        assert host.fb_disk_get_tiles(d.h, C.byref(cx), C.byref(ns)) == 0
        return ns.value
    assert get() == 0
    for want in (4, 8, 16, 0):
        d.check(host.fb_disk_set_tiles(d.h, 0, want))
        assert get() == want
        d.check(host.fb_disk_set_tiles(d.h, cx, ns))
        assert get() == want
    d.close()


@pytest.mark.parametrize("feel", [False, True])
@pytest.mark.parametrize("mesh", [(4, 4, 1), (4, 400, 1), (4, 4, 4), (4, 100, 100), (64, 12, 9)])
def test_params_bytes_is_an_upper_bound(host, mesh, feel):
    """What a disk requests stays within what fb_params_bytes says, with the
    scratch of planets that feel the disk too."""
    from fargo3d_b200 import Planet, _abi, config_fargo2d, config_p3disof
    cfg = config_fargo2d(*mesh[:2]) if mesh[2] == 1 else config_p3disof(*mesh)
    p = _abi.params_of(cfg.replace(planets=[Planet(1.0, 1e-3, True, True)]) if feel else cfg)
    for prec in (_abi.FB_FP64, _abi.FB_FP32):
        h, used, bound = C.c_void_p(), C.c_size_t(), C.c_size_t()
        assert host.fb_disk_create(C.byref(p), prec, 0, C.byref(h)) == 0
        assert host.fb_disk_bytes(h, C.byref(used)) == 0 and host.fb_params_bytes(C.byref(p), prec, C.byref(bound)) == 0
        assert used.value <= bound.value
        assert host.fb_disk_destroy(h) == 0
