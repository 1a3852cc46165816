"""2D solves of more sources than SMs at the widths where two of them still share
an SM and where they no longer do: the times at the receivers against the CPU
oracle (the same bound as for one source)."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_solver2d_diag import _model, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [321, 384, 385, 448, 449, 512])
def test_sources_sharing_an_sm(fk, nx):
    nz, h, ns = 31, 10.0, 160
    vel = _model(nz, nx, nx)
    rng = np.random.default_rng(nx)
    zs, xs = rng.uniform(0, (nz - 1) * h, ns), rng.uniform(0, (nx - 1) * h, ns)
    s = fk.fteik2d()
    s.initialize(nx, nz, h, h, nsweep=2, eps=5.0)
    s.setCellVelocityNatural(vel)
    s.setSources(xs, zs)
    zr, xr = np.zeros(9), np.linspace(0, (nx - 1) * h, 9)
    s.setReceivers(xr, zr)
    s.solveLSM()
    ttr = s.getTravelTimes()
    for k in (0, 80, 147, 148, 159):
        ref = _oracle(nz, nx, (h, h), vel, (zs[k], xs[k]), 5.0, 2)
        want, _ = O.receivers(False, (nz, nx, 1), (0, 0, 0), (h, h, 1.0), zr, xr, None, ref)
        assert np.max(np.abs(ttr[k] - want)) <= 1e-12 * np.max(want)
    s.free()
