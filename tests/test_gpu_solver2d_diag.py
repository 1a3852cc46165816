"""The diagonal 2D walk against the CPU oracle where it can go wrong: columns
around its warps and its limit (513 takes the walk in place), few rows, unequal
spacing, spherical regions smaller and larger than the table of near nodes,
sources in the corners and last cells, models whose roots leave the range of
the branch-free square root, and more sources than SMs."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def _model(nz, nx, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    vz = 3000.0 + 1000.0 * (np.arange(nz - 1) > 0.4 * nz)
    return (scale * vz[None, :] * (1.0 + 0.1 * rng.uniform(-1, 1, (nx - 1, nz - 1)))).ravel()


def _oracle(nz, nx, h, vel, src, eps, nsweep):
    si, sa = O.source_snap(False, (nz, nx, 1), (0, 0, 0), (h[0], h[1], 1.0), (src[0], src[1], 0.0))
    return O.solve2d((nz, nx), h, 1.0 / vel, si[:2], sa[:2], eps, nsweep)[0]


@pytest.mark.parametrize("nz,nx,h,eps,nsweep,scale", [
    (3, 3, (10.0, 10.0), 2.0, 2, 1.0), (5, 32, (10.0, 12.5), 5.0, 1, 1.0), (40, 33, (20.0, 10.0), 0.0, 2, 1.0),
    (65, 31, (10.0, 10.0), 9.0, 3, 1.0), (21, 64, (10.0, 10.0), 2.7, 0, 1.0), (50, 257, (5.0, 7.0), 5.0, 2, 1.0),
    (33, 320, (5.0, 5.0), 6.0, 2, 1.0), (20, 321, (5.0, 5.0), 5.0, 2, 1.0), (30, 512, (5.0, 5.0), 5.0, 2, 1.0),
    (30, 513, (5.0, 5.0), 5.0, 2, 1.0), (300, 40, (5.0, 5.0), 5.0, 2, 1.0), (40, 50, (10.0, 10.0), 5.0, 2, 1e105)])
@pytest.mark.parametrize("where", ["inside", "corner", "end"])
def test_matches_oracle(fk, nz, nx, h, eps, nsweep, scale, where):
    vel = _model(nz, nx, nz * 1000 + nx, scale)
    z, x = (nz - 1) * h[0], (nx - 1) * h[1]
    src = {"inside": (0.37 * z, 0.61 * x), "corner": (0.0, 0.0), "end": (z, x)}[where]
    s = fk.fteik2d()
    s.initialize(nx, nz, h[1], h[0], nsweep=nsweep, eps=eps)
    s.setCellVelocityNatural(vel)
    s.setSources(src[1], src[0])
    s.solveSourceLSM(1)
    tt = s.getTravelTimeField()
    ref = _oracle(nz, nx, h, vel, src, eps, nsweep)
    assert np.max(np.abs(tt - ref)) <= 1e-12 * np.max(ref)
    s.free()


@pytest.mark.parametrize("nx", [45, 300])
def test_more_sources_than_sms(fk, nx):
    nz, h, ns = 37, 10.0, 150
    vel = _model(nz, nx, 5)
    rng = np.random.default_rng(2)
    zs, xs = rng.uniform(0, (nz - 1) * h, ns), rng.uniform(0, (nx - 1) * h, ns)
    s = fk.fteik2d()
    s.initialize(nx, nz, h, h, nsweep=2, eps=5.0)
    s.setCellVelocityNatural(vel)
    s.setSources(xs, zs)
    zr, xr = np.zeros(9), np.linspace(0, (nx - 1) * h, 9)
    s.setReceivers(xr, zr)
    s.solveLSM()
    ttr = s.getTravelTimes()
    for k in (0, 1, 77, 148, 149):
        ref = _oracle(nz, nx, (h, h), vel, (zs[k], xs[k]), 5.0, 2)
        want, _ = O.receivers(False, (nz, nx, 1), (0, 0, 0), (h, h, 1.0), zr, xr, None, ref)
        assert np.max(np.abs(ttr[k] - want)) <= 1e-12 * np.max(want)
    s.free()
