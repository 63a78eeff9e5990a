"""The tile table and the tuner on a stand-in batch: a tuned column segment is
set whatever the table says of the azimuthal width, and the tuner's width does
not come from noise."""
import pytest


class _Batch:
    """Takes the tuner's calls; every profiled step gives another sweep_x time."""

    def __init__(self, cfgs, precision="fp32", device=0, tiles=None):
        self.cfgs, self.precision, self.set, self.steps = cfgs, precision, {}, 0

    def load_initial_states(self):
        pass

    def run(self, n):
        pass

    def close(self):
        pass

    def set_tiles(self, i, cx, ns):
        self.set[i] = (cx, ns)

    def tiles(self, i):
        return 4, 0

    def profile_step(self):
        self.steps += 1
        return {"sweep_x": 1.0 / self.steps, "sweep_cols": {4: 3.0, 8: 1.0, 16: 2.0}.get(self.set[0][1], 9.0)}


@pytest.mark.parametrize("width,want", [(4, 4), (0, 0), (16, 0), (5, 0)])   # 16 x 128: too much shared memory
def test_a_segment_is_set_with_any_width(width, want):
    from fargo3d_b200 import config_fargo2d
    from fargo3d_b200.autotune import TileTable, shape_key
    cfg = config_fargo2d(128, 64)
    t = TileTable({shape_key(cfg, "fp64"): {"sweep_x_cells": width, "col_segment": 8}})
    b = _Batch([cfg, config_fargo2d(96, 64)], "fp64")
    t.apply(b)
    assert b.set == {0: (want, 8)}
    assert t.tiles(cfg, "fp64") == (want, 8) and t.tiles(b.cfgs[1], "fp64") is None


def test_the_tuner_times_the_sweep_once(monkeypatch):
    import fargo3d_b200.batch
    from fargo3d_b200 import config_fargo2d
    from fargo3d_b200.autotune import cx_candidates, tune_shape
    monkeypatch.setattr(fargo3d_b200.batch, "Batch", _Batch)
    e = tune_shape(config_fargo2d(256, 128), "fp32", min_cells=1, reps=2)
    assert (e["sweep_x_cells"], e["col_segment"]) == (4, 8)   # the library's width, the fastest segment
    assert set(e["ms"]["sweep_x"]) == {str(c) for c in cx_candidates(256, "fp32")}
    assert len(set(e["ms"]["sweep_x"].values())) == 1
