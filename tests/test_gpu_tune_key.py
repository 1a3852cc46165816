"""The batch's tuning cache keeps the choices of different knob settings apart:
a search that a set knob limited decides nothing for an open one (which may take
the tile schedule), a set knob stays as set, and lines of the older six-value
form are searched again."""
import re

import numpy as np
import pytest

from models import layered_grf_cells

pytestmark = pytest.mark.gpu

OPEN = (-1, -1, -1, -1)


def _solve(fk, n, cfg):
    old = fk.set_slab_config(*cfg)
    try:
        b = fk.Batch3D([n + (25.0, 25.0, 25.0)], nsweep=2, eps=5.0, precision=4)
        b.setVelocityModel(1, layered_grf_cells(*n, seed=1, min_cells=2))
        b.setSources(1, *[np.array([0.4 * (m - 1) * 25.0]) for m in n])
        b.solve()
        c = b.slabConfig()
        b.finalize()
    finally:
        fk.set_slab_config(*old)
    return c


def _tiles(c):
    return c["tune_runs"] > 0 and c["init_ms"] == 0.0


def test_set_knobs_do_not_decide_for_open_ones(fk, monkeypatch, tmp_path):
    monkeypatch.setenv("FTEIK_B200_TUNE_CACHE", str(tmp_path / "t"))
    n = (31, 51, 43)                      # one source: the tiles take a third of the slabs' time
    c = _solve(fk, n, (0, 1, 8, -1))
    assert c["tune_runs"] > 0 and not _tiles(c)
    assert _tiles(_solve(fk, n, OPEN))
    assert _solve(fk, n, OPEN)["tune_runs"] == 0
    assert _solve(fk, n, (0, 1, 8, -1))["tune_runs"] == 0


def test_set_knobs_survive_a_hit(fk, monkeypatch, tmp_path):
    monkeypatch.setenv("FTEIK_B200_TUNE_CACHE", str(tmp_path / "t"))
    n = (29, 52, 45)
    _solve(fk, n, OPEN)
    for pairs, progress in ((0, 32), (1, 8), (0, 8), (1, 32)):
        for _ in range(2):                # searched, then from the cache
            c = _solve(fk, n, (-1, pairs, progress, -1))
            assert (c["pairs"], c["progress"]) == (pairs, progress)


def test_six_value_lines_are_searched_again(fk, monkeypatch, tmp_path):
    monkeypatch.setenv("FTEIK_B200_TUNE_CACHE", str(tmp_path / "t"))
    _solve(fk, (30, 50, 44), OPEN)
    line = (tmp_path / "t").read_text().split("\n")[0]
    key, values = line.split(" ", 1)
    key = re.sub(r"v7\|k[-0-9,]*\|", "", key.replace("30x50x44x1", "30x49x46x1"))
    (tmp_path / "t").write_text(" ".join([key] + values.split()[:6]) + "\n")
    assert _tiles(_solve(fk, (30, 49, 46), OPEN))
