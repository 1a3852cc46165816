"""Grid search with the misfit bounds.  L2 (many events): the optimum, origin
time and misfit are the full search's bit for bit; L1: the FP64 exhaustive
search's up to the FP32 ranking, whatever the bound rules out -- graded and skipped picks, tables with infinities, ties, grids around
the size and event count from which the bound is used, every table width."""
import numpy as np
import pytest

import oracle_lib as O
from models import station_tables, synthetic_events

pytestmark = pytest.mark.gpu


def _oracle(tables, picks, wts):
    tepoch = np.max(picks)
    use = wts > 0
    obs = np.where(use, (picks - tepoch).astype(np.float32), np.float32(0))
    obj, t0 = O.locate_l2_field(tables, obs, wts.astype(np.float32), (~use).astype(np.uint8))
    g = np.nanargmin(obj)         # MINLOC: the first minimum, undefined misfits (an unreachable table) aside
    return g + 1, float(t0[g]) + tepoch, float(obj[g])


@pytest.mark.parametrize("ntf,nz,nx,ny,nev", [(1, 16, 17, 16, 8), (3, 16, 16, 16, 9), (16, 17, 16, 16, 8),
                                              (17, 21, 19, 23, 33), (33, 16, 16, 16, 7), (64, 25, 31, 29, 40)])
@pytest.mark.parametrize("kind", ["times", "random", "ties"])
def test_bounded_search_matches_oracle_bitwise(fk, ntf, nz, nx, ny, nev, kind):
    ngrd = nz * nx * ny
    rng = np.random.default_rng(ntf * 100 + nev)
    if kind == "times":
        tables = station_tables(nz, nx, ny, 100.0, ntf, seed=ntf)
    elif kind == "random":
        tables = rng.uniform(0.5, 12.0, (ntf, ngrd)).astype(np.float32)
    else:                         # repeated columns: first index wins
        tables = np.tile(rng.uniform(0.5, 3.0, (ntf, ngrd // 4 + 1)).astype(np.float32), (1, 4))[:, :ngrd].copy()
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
    oi, t0, ob = loc.locateEvents(np.arange(1, nev + 1))
    for e in range(nev):
        want = _oracle(tables, picks[e], wts[e])
        assert (oi[e], t0[e], ob[e]) == want, e
    loc.finalize()


@pytest.mark.parametrize("ntf,nz,nx,ny,nev", [(1, 16, 17, 16, 3), (2, 16, 16, 16, 17), (16, 17, 16, 16, 8),
                                              (17, 21, 19, 23, 33), (45, 16, 16, 15, 7), (64, 25, 31, 29, 20)])
@pytest.mark.parametrize("kind", ["times", "random"])
def test_bounded_l1_matches_fp64_exhaustive(fk, ntf, nz, nx, ny, nev, kind):
    ngrd = nz * nx * ny
    rng = np.random.default_rng(ntf * 10 + nev)
    if kind == "times":
        tables = station_tables(nz, nx, ny, 100.0, ntf, seed=ntf)
    else:
        tables = rng.uniform(0.5, 12.0, (ntf, ngrd)).astype(np.float32)
    _, picks = synthetic_events(tables, nev, seed=ntf + 2)
    wts = np.full(picks.shape, 0.5)
    wts[rng.random(picks.shape) < 0.15] = 0.0
    wts[:, 0] = 0.5
    loc = fk.Locator(nev, ntf, ngrd)
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    loc.setNorm(1)
    oi, t0, ob = loc.locateEvents(np.arange(1, nev + 1))
    for e in range(nev):
        red = picks[e] - picks[e].max()
        _, _, gob = O.locate_l1_best64(tables, red, wts[e])
        _, t_here, ob_here = O.locate_l1_best64(tables[:, [oi[e] - 1]], red, wts[e])
        # the FP32 ranking misfit is off by at most (N + 1) 2^-24 sum (|o| + |T|), both points
        off = 2 * 65 * 2.0 ** -24 * 0.5 * (np.abs(red).sum() + np.abs(tables).max(1).sum())
        assert ob_here <= gob + off, (e, ob_here, gob)
        assert abs(ob[e] - ob_here) <= 1e-9 * max(ob_here, 1e-12)
        assert abs(t0[e] - (t_here + picks[e].max())) <= 1e-9 * max(1.0, abs(t0[e]))
    loc.finalize()
