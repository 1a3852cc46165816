"""Waits that run out, on each of the 3D schedules (the slabs with a knob set, the
tiles with all knobs open): the solve returns an error, the next one with the
default limit the right field -- one source in both precisions, and a batch
iterated to convergence, whose tiles also wait for one another after each pass."""
import numpy as np
import pytest

from models import layered_grf_cells
from test_gpu_tiles import H, SLABS, TILES, _cells, _solve, _src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [SLABS, TILES], ids=["slabs", "tiles"])
@pytest.mark.parametrize("precision", [4, 8])
def test_single_source(fk, cfg, precision):
    n = (40, 70, 64)
    vel, src = _cells(n, 7), _src(n, "inside")
    want = _solve(fk, n, vel, src, cfg, precision)
    old = fk.set_spin_limit(0)
    try:
        for _ in range(3):
            with pytest.raises(fk.FteikError):
                _solve(fk, n, vel, src, cfg, precision)
    finally:
        fk.set_spin_limit(old)
    assert np.array_equal(_solve(fk, n, vel, src, cfg, precision), want)


@pytest.mark.parametrize("cfg", [SLABS, TILES], ids=["slabs", "tiles"])
def test_converged_batch(fk, cfg):
    n = (31, 53, 42)                      # one source: the tuner takes the tiles by a factor of three
    old = fk.set_slab_config(*cfg)
    try:
        b = fk.Batch3D([n + H], eps=5.0, precision=4, convTol=0.0, maxPass=20)
        b.setVelocityModel(1, layered_grf_cells(*n, seed=2, min_cells=2))
        b.setSources(1, *[np.array([v]) for v in _src(n, "inside")])
        b.solve()
        c = b.slabConfig()
        assert (c["tune_runs"] > 0 and c["init_ms"] == 0.0) == (cfg == TILES)
        want, info = b.fields32(1).copy(), b.solveInfo(1, 1)
        spin = fk.set_spin_limit(0)
        try:
            for _ in range(3):
                with pytest.raises(fk.FteikError):
                    b.solve()
        finally:
            fk.set_spin_limit(spin)
        b.solve()
        assert np.array_equal(b.fields32(1), want) and b.solveInfo(1, 1) == info
        b.finalize()
    finally:
        fk.set_slab_config(*old)
