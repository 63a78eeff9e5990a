"""The azimuthal sweep's strips: rings at, below and above the widths a warp
writes (52 cells in FP64, 116 in FP32) and the whole-ring strips (64, 128),
odd rings (plain loads), rings of several strips from staged pieces, marches of
one ring to eight with a remainder, shifts beyond a ring, fused new velocities
and damping, against the oracle: FP64 bit for bit, FP32 to 1e-5 relative L1
density after 3 steps (the FP32 path's stated bound) and 3e-5 relative L1
velocities (some 30 FP32 roundings of 6e-8 of the terms of a step, whose
largest are a few times the radial velocity of these states)."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def _cfg(nx, ny, **kw):
    from fargo3d_b200 import config_fargo2d
    return config_fargo2d(nx, ny, seed=31 + nx).replace(noise=0.05, **kw)


def _near(got, want, cfg):
    for k in ("rho", "vx", "vy") + (("vz",) if cfg.is3d else ()):
        w = want[k].reshape(got[k].shape)
        assert np.abs(got[k] - w).sum() <= (1e-5 if k == "rho" else 3e-5) * np.abs(w).sum(), k


def _check(cfg, steps=3):
    import pyoracle
    from fargo3d_b200 import Batch, Disk, initial_state
    pyoracle.build()
    init = [initial_state(cfg)]
    want, dts, _ = pyoracle.run(cfg, steps, "oracle", state=init)
    d = Disk(cfg, "fp64")
    d.set_state(*init[0])
    d.initialize()
    assert np.array_equal(d.run(steps), dts)
    got = d.state()
    d.close()
    for k in ("rho", "vx", "vy") + (("vz",) if cfg.is3d else ()):
        assert np.array_equal(got[k], want[0][k].reshape(got[k].shape)), k
    if cfg.adiabatic:
        return
    b = Batch([cfg, cfg], "fp32")
    for i in range(2):
        b.set_state(i, *init[0])
    b.initialize()
    b.run(steps)
    for i in range(2):
        _near(b.state(i), want[0], cfg)
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [8, 17, 51, 52, 53, 64, 66, 104, 112, 116, 120, 128, 129, 232, 236, 250, 255, 260])
def test_ring_lengths(nx):
    _check(_cfg(nx, 11))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(64, 4), (60, 5), (52, 6), (128, 7), (100, 200)])
def test_row_counts(nx, ny):
    """From four rows, of which some mirror to both radial sides' ghosts."""
    _check(_cfg(nx, ny))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx", [52, 120, 232, 250, 260])
@pytest.mark.parametrize("rows", [3, 8])
def test_long_marches(nx, rows, precision):
    """A batch with enough strips for marches of `rows` rings (two times the
    chip's 148 x 16 warps each) over 301 rows, which no march length divides;
    the source stage and the column sweeps march 3 to 16 rows with them."""
    import pyoracle
    from fargo3d_b200 import Batch, initial_state
    pyoracle.build()
    cfg = _cfg(nx, 301)
    init = [initial_state(cfg)]
    want, _, _ = pyoracle.run(cfg, 3, "oracle", state=init)
    width = 52 if precision == "fp64" else 116
    copies = -(-rows * 148 * 16 * 2 // (-(-nx // width) * 301))
    b = Batch([cfg] * copies, precision)
    b.set_states(init * copies)
    b.initialize()
    b.run(3)
    for i in (0, copies - 1):
        got = b.state(i)
        if precision == "fp32":
            _near(got, want[0], cfg)
            continue
        for k in ("rho", "vx", "vy"):   # a batch's planets move to the last bits differently
            w = want[0][k].reshape(got[k].shape)
            assert np.abs(got[k] - w).max() <= 1e-10 * np.abs(w).max(), k
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("omega", [-60.0, 0.0, 60.0])
def test_shifts_beyond_the_ring(omega):
    """A fast frame: rings shift by more cells than they hold, either way."""
    _check(_cfg(24, 12, frame="F", omegaframe=omega), steps=2)


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [48, 65])
def test_adiabatic_energy(nx):
    from fargo3d_b200 import config_adiabatic2d
    _check(config_adiabatic2d(nx, 13, seed=5))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz", [(52, 5), (64, 4), (75, 6)])
def test_3d(nx, nz):
    from fargo3d_b200 import config_p3disof
    _check(config_p3disof(nx, 10, nz, seed=3), steps=2)
