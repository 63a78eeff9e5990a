"""The one-disk step's parts go out as launches first and as captured graphs
later: the same bits across the change, and what the capture holds -- tiles,
the planets, the frame, two disks on their own threads -- stays current."""
import os
import sys
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def _cfg(feel=False, seed=4):
    from fargo3d_b200 import Planet, config_fargo2d
    c = config_fargo2d(48, 20, seed=seed).replace(noise=0.02)
    return c.replace(frame="F", omegaframe=1.0, planets=[Planet(1.0, 1e-3, True, False)]) if feel else c


@pytest.mark.gpu
@pytest.mark.parametrize("feel", [False, True])
def test_steps_match_the_oracle_across_the_capture(feel):
    import pyoracle
    from fargo3d_b200 import Disk, initial_state
    pyoracle.build()
    cfg = _cfg(feel)
    init = initial_state(cfg)
    want, dts, sc = pyoracle.run(cfg, 12, "oracle", state=[init])
    d = Disk(cfg, "fp64")
    d.set_state(*init)
    d.initialize()
    got = d.run(7)
    d.set_state(**dict(zip(("rho", "vx", "vy", "vz", "cs"), [d.state()[k] for k in ("rho", "vx", "vy", "vz")] + [init[4]])))
    assert np.array_equal(np.concatenate([got, d.run(5)]), dts)   # the state set again between steps
    st = d.state()
    for k in ("rho", "vx", "vy"):
        assert np.array_equal(st[k], want[0][k].reshape(st[k].shape)), k
    assert np.array_equal(d.scalars(), sc)
    d.close()


@pytest.mark.gpu
def test_step_in_parts_and_whole_agree():
    from fargo3d_b200 import Disk
    a, b = Disk(_cfg(), "fp64"), Disk(_cfg(), "fp64")
    for d in (a, b):
        d.load_initial_state()
    for n in range(10):
        dt = a.step()
        if n % 3 == 2:
            assert b.step() == dt
        else:
            assert b.step_advance(1e30, b.step_begin()) == dt
            b.step_transport()
    for k in ("rho", "vx", "vy"):
        assert np.array_equal(a.state()[k], b.state()[k])
    a.close()
    b.close()


@pytest.mark.gpu
def test_changed_tiles_and_threads():
    from fargo3d_b200 import Disk, _abi
    ref = {}
    for seed in (4, 5):
        d = Disk(_cfg(seed=seed), "fp64")
        d.load_initial_state()
        d.run(12)
        ref[seed] = d.state()
        d.close()
    out = {}

    def work(seed):
        d = Disk(_cfg(seed=seed), "fp64")
        d.load_initial_state()
        d.run(6)
        _abi.check(_abi.lib().fb_disk_set_tiles(d._h, 0, 8))
        d.run(6)
        out[seed] = d.state()
        d.close()

    ts = [threading.Thread(target=work, args=(s,)) for s in (4, 5)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for seed in (4, 5):
        for k in ("rho", "vx", "vy"):
            assert np.array_equal(out[seed][k], ref[seed][k])


@pytest.mark.gpu
def test_advances_without_a_begin():
    """A whole step and then advances with the caller's own CFL minimum: the
    same bits whether or not the stream is waited for between the calls."""
    from fargo3d_b200 import Disk
    got = []
    for wait in (True, False):
        d = Disk(_cfg(), "fp64")
        d.load_initial_state()
        dts = []
        for n in range(8):
            dts.append(d.step())
            if wait:
                d.state()
            dts.append(d.step_advance(1e30, 0.5 * dts[-1]))
            if wait:
                d.state()
            d.step_transport()
        got.append((dts, d.state()))
        d.close()
    assert got[0][0] == got[1][0]
    for k in ("rho", "vx", "vy"):
        assert np.array_equal(got[0][1][k], got[1][1][k]), k


@pytest.mark.gpu
def test_members_of_a_batch_on_their_own_threads():
    """Members share the batch's stream: parts captured by one thread hold
    nothing of what the other queues meanwhile."""
    import ctypes as C
    from fargo3d_b200 import Batch, Disk, _abi
    ref = {}
    for seed in (4, 5):
        d = Disk(_cfg(seed=seed), "fp64")
        d.load_initial_state()
        ref[seed] = (d.run(40), d.state())
        d.close()
    b = Batch([_cfg(seed=4), _cfg(seed=5)], "fp64")
    b.load_initial_states()
    b.sync()
    dts = {}

    def work(i):
        dt = C.c_double()
        dts[4 + i] = []
        for _ in range(40):
            _abi.check(_abi.lib().fb_disk_step(b._members[i]._h, 1e30, C.byref(dt)))
            dts[4 + i].append(dt.value)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for i, seed in enumerate((4, 5)):
        assert dts[seed] == ref[seed][0]
        st = b.state(i)
        for k in ("rho", "vx", "vy"):
            assert np.array_equal(st[k], ref[seed][1][k]), (seed, k)
    b.close()


@pytest.mark.gpu
def test_transport_inside_a_callers_capture():
    import torch
    from fargo3d_b200 import Disk
    a, b = Disk(_cfg(), "fp64"), Disk(_cfg(), "fp64")
    for d in (a, b):
        d.load_initial_state()
        for _ in range(6):   # the parts go out as graphs by now
            d.step_advance(1e30, d.step_begin())
            d.step_transport()
        d.step_advance(1e30, d.step_begin())
    a.step_transport()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.ExternalStream(b.stream)):
        g.capture_begin(capture_error_mode="thread_local")
        b.step_transport()
        g.capture_end()
        g.replay()
    for k in ("rho", "vx", "vy"):
        assert np.array_equal(a.state()[k], b.state()[k]), k
    assert a.step() == b.step()
    del g
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,kind", [("fp32", "2d"), ("fp32", "3d"), ("fp64", "3d"), ("fp64", "adiabatic"),
                                            ("fp64", "dust"), ("fp64", "diffusion"), ("fp32", "dust")])
def test_captured_parts_are_the_launches(precision, kind):
    """The same bits from launches (a profiled disk's steps) and from graphs,
    of every kind of step."""
    from fargo3d_b200 import Disk, _abi, config_adiabatic2d, config_multifluid, config_p3disof
    cfg = {"2d": lambda: _cfg(True), "3d": lambda: config_p3disof(36, 12, 6, seed=2),
           "adiabatic": lambda: config_adiabatic2d(48, 20, seed=2), "dust": lambda: config_multifluid(48, 20, nfluids=4),
           "diffusion": lambda: config_multifluid(48, 20, nfluids=3, dust_diffusion=True)}[kind]().replace(noise=0.02)
    got = []
    for eager in (1, 0):
        d = Disk(cfg, precision)
        d.load_initial_state()
        _abi.lib().fb_disk_profile(d._h, eager)
        got.append((d.run(12), [d.state(f) for f in range(cfg.nfluids)]))
        d.close()
    assert got[0][0] == got[1][0]
    for a, b in zip(got[0][1], got[1][1]):
        for k in ("rho", "vx", "vy", "vz"):
            assert np.array_equal(a[k], b[k]), k
