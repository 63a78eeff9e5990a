"""The marching column sweeps: segment lengths that do and do not divide the
rows, the default length from the mesh's size and every set tile, 2D and 3D
(two groups of quantities), FP64 bit for bit against the oracle, FP32 against
FP64 to 1e-5 relative L1 density."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz", [(32, 4, 1), (33, 7, 1), (129, 63, 1), (16, 900, 1), (20, 5, 4), (33, 10, 7)])
@pytest.mark.parametrize("tile", [0, 4, 8, 16])
def test_segments(nx, ny, nz, tile):
    import pyoracle
    from fargo3d_b200 import Disk, _abi, config_fargo2d, config_p3disof, initial_state
    pyoracle.build()
    cfg = (config_fargo2d(nx, ny, seed=3) if nz == 1 else config_p3disof(nx, ny, nz, seed=3)).replace(noise=0.05)
    init = initial_state(cfg)
    want, dts, _ = pyoracle.run(cfg, 2, "oracle", state=[init])
    keys = ("rho", "vx", "vy") + (("vz",) if nz > 1 else ())
    for prec in ("fp64", "fp32"):
        d = Disk(cfg, prec, tiles=None)
        _abi.check(_abi.lib().fb_disk_set_tiles(d._h, 0, tile))
        d.set_state(*init)
        d.initialize()
        got_dt = d.run(2)
        got = d.state()
        d.close()
        if prec == "fp64":
            assert np.array_equal(got_dt, dts)
            for k in keys:
                assert np.array_equal(got[k], want[0][k].reshape(got[k].shape)), k
        else:
            w = want[0]["rho"].reshape(got["rho"].shape)
            assert np.abs(got["rho"] - w).sum() <= 1e-5 * np.abs(w).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nz", [(8, 20000, 1), (4, 4, 8200)])
def test_segments_and_layers_of_eight_fluids_beyond_a_grid(nx, ny, nz, prec):
    """Long thin meshes of many fluids: segments x fluids (2D, two rows each)
    and layers x fluids (3D) are more than a grid's third index takes."""
    import pyoracle
    from fargo3d_b200 import Disk, config_multifluid, config_p3disof, initial_state
    pyoracle.build()
    inv = (100.0, 30.0, 10.0, 3.0, 1.0, 0.3, 0.1)
    cfg = (config_multifluid(nx, ny, nfluids=8, invstokes=inv, seed=2) if nz == 1 else
           config_p3disof(nx, ny, nz, seed=2).replace(nfluids=8, invstokes=inv))
    init = [initial_state(cfg, f) for f in range(8)]
    want, dts, _ = pyoracle.run(cfg, 2, "oracle", state=init)
    d = Disk(cfg, prec)
    for f in range(8):
        d.set_state(*init[f], fluid=f)
    d.initialize()
    got_dt = d.run(2)
    for f in range(8):
        r = d.state(f)["rho"]
        w = want[f]["rho"].reshape(r.shape)
        if prec == "fp64":
            assert np.array_equal(got_dt, dts) and np.array_equal(r, w), f
        else:
            assert np.abs(r - w).sum() <= 1e-5 * np.abs(w).sum(), f
    d.close()
