"""The allocation-free grid search on grids as large as an index holds (two tables of
2^31 - 129 points), against the objective evaluated in torch piece by piece."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_points_up_to_the_index_limit(fk):
    import torch
    ngrd, ntf, nev = (1 << 31) - 129, 2, 8
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    tables = torch.empty(ntf, ngrd, dtype=torch.float32, device=dev)
    for i in range(ntf):
        tables[i].uniform_(1.0, 9.0, generator=g)
    rng = np.random.default_rng(2)
    obs = rng.uniform(-0.5, 0.5, (nev, ntf)).astype(np.float32)
    tables[0, -50] = 100.0
    obs[0] = (100.0 + 1.0, float(tables[1, -50]) + 1.0)
    tables[0, -1] = -100.0
    obs[1] = (-100.0 + 2.0, float(tables[1, -1]) + 2.0)
    o = torch.from_numpy(obs).to(dev)
    w = torch.ones(nev, ntf, dtype=torch.float32, device=dev)
    out = torch.full((nev,), -1, dtype=torch.int32, device=dev)
    t0 = torch.zeros(nev, dtype=torch.float32, device=dev)
    obj = torch.zeros(nev, dtype=torch.float32, device=dev)
    torch.cuda.synchronize()
    ierr = ctypes.c_int(1)
    fk.lib().fteik_b200_locate_l2_noalloc(ngrd, ngrd, ntf, ctypes.c_void_p(tables.data_ptr()), nev,
                                          ctypes.c_void_p(o.data_ptr()), ctypes.c_void_p(w.data_ptr()),
                                          ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(t0.data_ptr()),
                                          ctypes.c_void_p(obj.data_ptr()), None, ctypes.byref(ierr))
    torch.cuda.synchronize()
    assert ierr.value == 0
    half = torch.tensor(0.70710677, dtype=torch.float32, device=dev)
    for e in range(nev):
        best = (float("inf"), -1)
        for p0 in range(0, ngrd, 1 << 28):
            T = tables[:, p0:p0 + (1 << 28)]
            t = (o[e, 0] - T[0]) * 0.5 + (o[e, 1] - T[1]) * 0.5
            a, b = half * (o[e, 0] - (T[0] + t)), half * (o[e, 1] - (T[1] + t))
            f = a * a + b * b
            m = float(f.min())
            if m < best[0]:
                best = (m, p0 + int((f == m).nonzero()[0, 0]))
        assert (float(obj[e]), int(out[e])) == best, e
    assert out[:2].tolist() == [ngrd - 50, ngrd - 1]
    del tables, T, t, a, b, f
    torch.cuda.empty_cache()
