"""Grid search with weights whose squares, or whose products with the misfits, leave
the range of normal FP32 numbers: the bounds may then rule nothing out, and the
optimum is still the full search's -- the oracle's, bit for bit (L2), or the first
minimum of the FP32 misfits formed as in the search (L1)."""
import numpy as np
import pytest

from models import station_tables, synthetic_events
from test_gpu_locate_bound import _oracle

pytestmark = pytest.mark.gpu


def _locate(fk, tables, picks, wts, norm):
    nev, ntf = picks.shape
    loc = fk.Locator(nev, ntf, tables.shape[1])
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    loc.setNorm(norm)
    got = [np.array(v) for v in loc.locateEvents(np.arange(1, nev + 1))]
    loc.finalize()
    return got


def _tables(ntf, ngrd):
    return np.ascontiguousarray(station_tables(64, 64, ngrd // 4096 + 1, 50.0, ntf, seed=ntf)[:, :ngrd])


@pytest.mark.parametrize("scale", [1e-24, 1e-23, 1e-22, 1e-21, 1e-20, 1e-18, 1e-12, 1e12, 1e18, 1e19])
@pytest.mark.parametrize("ntf,ngrd,nev", [(1, 4100, 9), (5, 9000, 12), (20, 9000, 12), (20, (1 << 18) + 5, 192)])
def test_l2_weights_of_any_size(fk, scale, ntf, ngrd, nev):
    tables = _tables(ntf, ngrd)
    _, picks = synthetic_events(tables, nev, seed=ntf + 1)
    rng = np.random.default_rng(ntf)
    wts = scale * rng.choice([1.0, 0.75, 0.5, 0.25], picks.shape)
    got = _locate(fk, tables, picks, wts, 2)
    for e in range(0, nev, 1 if nev < 20 else 37):
        assert tuple(v[e] for v in got) == _oracle(tables, picks[e], wts[e]), e

def _l1_best(tables, picks, w):
    r = np.sort((picks - picks.max()).astype(np.float32)[:, None] - tables, axis=0)
    n = len(r)
    obj = np.zeros(tables.shape[1], np.float32)
    for i in range(n):
        if i < n // 2:
            obj = obj - r[i]
        elif i >= n - n // 2:
            obj = obj + r[i]
    key = (obj * np.float32(w)).view(np.uint32)      # ordered as the search orders them
    return int(np.argmin(key)) + 1


@pytest.mark.parametrize("scale", [1e-44, 1e-42, 1e-40, 1e-38, 1e-30, 1e30, 1e37])
@pytest.mark.parametrize("ntf,ngrd,nev", [(5, 9000, 12), (20, 9000, 12), (20, (1 << 16) + 5, 40)])
def test_l1_weights_of_any_size(fk, scale, ntf, ngrd, nev):
    tables = _tables(ntf, ngrd)
    _, picks = synthetic_events(tables, nev, seed=ntf + 1)
    got = _locate(fk, tables, picks, np.full(picks.shape, scale), 1)
    for e in range(0, nev, 1 if nev < 20 else 7):
        assert got[0][e] == _l1_best(tables, picks[e], scale), e


@pytest.mark.parametrize("ngrd", [100, 5000])
def test_l1_weights_that_vanish_in_fp32(fk, ngrd):
    """Every ranked misfit is zero: the first point, with its FP64 values."""
    tables = _tables(7, ngrd)
    _, picks = synthetic_events(tables, 3, seed=5)
    w = 1e-50
    idx, t0, obj = _locate(fk, tables, picks, np.full(picks.shape, w), 1)
    r = picks - tables[:, 0].astype(np.float64)
    med = np.median(r, axis=1)
    assert (idx == 1).all()
    assert np.allclose(t0, med, rtol=1e-12, atol=1e-9)
    assert np.allclose(obj / w, np.abs(r - med[:, None]).sum(1), rtol=1e-9)
