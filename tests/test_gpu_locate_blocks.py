"""Grid search of many events on fine grids, bounded by blocks of 32 points: the
optimum, origin time and misfit equal, bit for bit, those of the same events
searched in smaller groups (each point bounded by itself) and the oracle's, at
the edges of blocks, of a thread block's 1024 points, of the table widths and of
the event groups.  L1: equal to the search in smaller groups."""
import numpy as np
import pytest

from models import station_tables, synthetic_events
from test_gpu_locate_bound import _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntf,ngrd,nev", [(1, 1 << 18, 192), (16, (1 << 18) + 1, 193), (17, (1 << 18) + 33, 256),
                                          (48, (1 << 18) + 1023, 257), (49, 1 << 19, 320), (64, (1 << 19) + 17, 200)])
@pytest.mark.parametrize("kind", ["times", "random"])
def test_blocks_match_points_and_oracle_bitwise(fk, ntf, ngrd, nev, kind):
    rng = np.random.default_rng(ntf + nev)
    if kind == "times":
        n = 64 * 64 * (ngrd // 4096 + 1)
        tables = np.ascontiguousarray(station_tables(64, 64, n // 4096, 50.0, ntf, seed=ntf)[:, :ngrd])
    else:
        tables = rng.uniform(0.5, 12.0, (ntf, ngrd)).astype(np.float32)
    _, picks = synthetic_events(tables, nev, seed=ntf + 1)
    wts = rng.choice([1.0, 0.75, 0.5, 0.25], picks.shape)
    wts[rng.random(picks.shape) < 0.15] = 0.0
    wts[:, 0] = 1.0
    if ntf > 3:                   # an unreachable table, unused by most events
        tables[2, : ngrd // 2] = np.inf
        wts[1:, 2] = 0.0
    loc = fk.Locator(nev, ntf, ngrd)
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    got = [np.array(v) for v in loc.locateEvents(np.arange(1, nev + 1))]
    for e0 in range(0, nev, 150):
        few = loc.locateEvents(np.arange(e0 + 1, min(nev, e0 + 150) + 1))
        for a, b in zip(got, few):
            np.testing.assert_array_equal(a[e0:e0 + 150], np.array(b))
    for e in (0, nev // 2, nev - 1):
        assert tuple(v[e] for v in got) == _oracle(tables, picks[e], wts[e]), e
    loc.finalize()


@pytest.mark.parametrize("ntf,ngrd,nev", [(1, 1 << 16, 32), (2, (1 << 16) + 1, 33), (17, (1 << 16) + 1055, 64), (32, 1 << 16, 300),
                                          (33, 1 << 18, 64), (64, (1 << 18) + 31, 65)])
@pytest.mark.parametrize("kind", ["times", "random"])
def test_l1_blocks_match_points(fk, ntf, ngrd, nev, kind):
    rng = np.random.default_rng(ntf * 10 + nev)
    if kind == "times":
        n = ngrd // 4096 + 1
        tables = np.ascontiguousarray(station_tables(64, 64, n, 50.0, ntf, seed=ntf)[:, :ngrd])
    else:
        tables = rng.uniform(0.5, 12.0, (ntf, ngrd)).astype(np.float32)
    _, picks = synthetic_events(tables, nev, seed=ntf + 2)
    wts = np.full(picks.shape, 0.5)
    wts[rng.random(picks.shape) < 0.15] = 0.0
    wts[:, 0] = 0.5
    if ntf > 3:                   # an unreachable table, unused by all events
        tables[2, : ngrd // 2] = np.inf
        wts[:, 2] = 0.0
    loc = fk.Locator(nev, ntf, ngrd)
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    loc.setNorm(1)
    got = [np.array(v) for v in loc.locateEvents(np.arange(1, nev + 1))]
    for e0 in range(0, nev, 30):
        few = loc.locateEvents(np.arange(e0 + 1, min(nev, e0 + 30) + 1))
        for a, b in zip(got, few):
            np.testing.assert_array_equal(a[e0:e0 + 30], np.array(b))
    loc.finalize()


@pytest.mark.parametrize("ntf", [15, 16, 32, 47, 48])
@pytest.mark.parametrize("nev,ngrd", [(1, 4111), (8, 4096), (21, 4225)])
def test_table_widths_match_oracle_bitwise(fk, ntf, nev, ngrd):
    tables = np.ascontiguousarray(station_tables(16, 16, 17, 100.0, ntf, seed=ntf)[:, :ngrd])
    _, picks = synthetic_events(tables, nev, seed=ntf + 1)
    rng = np.random.default_rng(ntf + nev)
    wts = rng.choice([1.0, 0.75, 0.5, 0.25], picks.shape)
    wts[rng.random(picks.shape) < 0.15] = 0.0
    wts[:, 0] = 1.0
    loc = fk.Locator(nev, ntf, tables.shape[1])
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    got = loc.locateEvents(np.arange(1, nev + 1))
    for e in range(nev):
        assert tuple(v[e] for v in got) == _oracle(tables, picks[e], wts[e]), e
    loc.finalize()
