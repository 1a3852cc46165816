"""Surrogate-pruned search over block shapes (node counts that are no multiple
of 4, below and above the 64 nodes of one load, blocks that stick out of the
grid), station counts odd and even and magnitudes that strain the FP32
screening: the result is a minimum of the FP64 misfit over its 26 neighbours
and its values are the FP64 ones."""
import numpy as np
import pytest

from models import linear_gradient_tables, synthetic_events

pytestmark = pytest.mark.gpu

N = (22, 30, 27)
H = 100.0


@pytest.mark.parametrize("ntf,shift", [(64, 0.0), (37, 0.0), (10, 3000.0)])
@pytest.mark.parametrize("block", [(4, 4, 4), (3, 3, 3), (5, 2, 1), (7, 4, 3), (8, 8, 8)])
def test_pruned_is_a_local_minimum(fk, ntf, shift, block):
    nz, nx, ny = N
    tables, sta = linear_gradient_tables(nz, nx, ny, H, ntf, seed=ntf)
    _, picks = synthetic_events(tables, 150, seed=3)
    tables = tables + np.float32(shift)      # a common delay: the same hypocentres, larger residuals
    nev = picks.shape[0]
    loc = fk.Locator(nev, ntf, tables.shape[1])
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], np.full(ntf, 0.5))
    loc.setGeometry(nz, nx, ny, H, H, H, *sta)
    fk.MLP(256, 5, seed=7)
    loc.trainSurrogate(nsamples=200_000, steps=600, batch=4096, lr=2e-3, vref=3000.0, seed=7)
    loc.buildSurrogate(block)
    loc.setMethod(2)
    oi, t0, ob = loc.locateEvents(np.arange(1, nev + 1))
    nodes = np.arange(tables.shape[1]).reshape(ny, nx, nz)
    for e in range(nev):
        red = picks[e] - picks[e].max()
        g = oi[e] - 1
        z, x, y = g % nz, g // nz % nx, g // (nz * nx)
        near = nodes[max(y - 1, 0):y + 2, max(x - 1, 0):x + 2, max(z - 1, 0):z + 2].ravel()
        d = red[:, None] - tables[:, near].astype(np.float64)
        obj = 0.5 * 0.25 * ((d - d.mean(0)) ** 2).sum(0)
        here = obj[near == g][0]
        # misfit64's one-pass sums cancel to about (n d^2) 2^-53 (1e-9 at 3000 s)
        tol = 1e-9 * here + 16 * 2.0 ** -53 * 0.25 * (red[:, None] - tables[:, [g]].astype(np.float64)).__pow__(2).sum()
        assert abs(ob[e] - here) <= tol and here <= obj.min() + 2 * tol, (e, here, obj.min())
    loc.finalize()
