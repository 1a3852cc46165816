"""The tile kernel shared by a batch's captured graph and a single-source solver of
other depths: deep and shallow solves in turn, each with the field it gave alone."""
import numpy as np
import pytest

from test_gpu_tiles import H, TILES, _cells, _solve, _src

pytestmark = pytest.mark.gpu


def test_solver_between_two_launches_of_a_batch(fk):
    n = (90, 64, 62)                      # 105 KB of shared memory a tile
    small = [(9, 33, 20), (5, 17, 9), (61, 20, 31), (160, 16, 16)]
    want = {m: _solve(fk, m, _cells(m, 3), _src(m, "inside"), TILES, 4) for m in small}
    b = fk.Batch3D([n + H], nsweep=2, eps=5.0, precision=4)
    b.setVelocityModel(1, _cells(n, 8))
    b.setSources(1, *[np.array([v]) for v in _src(n, "inside")])
    b.solve()
    assert b.slabConfig()["init_ms"] == 0.0          # the tiles
    field = b.fields32(1).copy()
    for m in small:
        assert np.array_equal(_solve(fk, m, _cells(m, 3), _src(m, "inside"), TILES, 4), want[m])
        b.solve()
        assert np.array_equal(b.fields32(1), field)
    b.finalize()
