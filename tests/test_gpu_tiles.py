"""The tile schedule of the 3D solve (taken where a solve's tiles fit the chip
and the launch configuration is left to the library) against the slab schedule
(a knob set): FP32 fields bit for bit, FP64 fields against the CPU oracle --
grids around the tile's 16 x 8 columns, sources in corners, faces and last
cells, spherical regions of no and of many cells, no passes, convergence, and
work lists that take several launches."""
import numpy as np
import pytest

import oracle_lib as O
from models import layered_grf_cells

pytestmark = pytest.mark.gpu

H = (25.0, 20.0, 30.0)
SLABS, TILES = (0, 0, 0, 0), (-1, -1, -1, -1)


def _cells(n, seed):
    rng = np.random.default_rng(seed)
    nz, nx, ny = n
    vz = 3000.0 + 1500.0 * (np.arange(nz - 1) > 0.4 * nz)
    return vz * (1.0 + 0.1 * rng.uniform(-1, 1, (ny - 1, nx - 1, nz - 1)))


def _solve(fk, n, vel, src, cfg, precision, nsweep=2, eps=5.0):
    old = fk.set_slab_config(*cfg)
    try:
        s = fk.fteik3d()
        s.initialize(n[1], n[2], n[0], H[1], H[2], H[0], nsweep=nsweep, eps=eps, precision=precision)
        s.setCellSlownessNatural(vel)
        s.setSources(src[1], src[2], src[0])
        s.solveSourceLSM(1)
        tt = s.getTravelTimeField()
        s.free()
    finally:
        fk.set_slab_config(*old)
    return tt


def _src(n, where):
    f = {"inside": (0.31, 0.57, 0.66), "corner": (0.0, 0.0, 0.0), "end": (1.0, 1.0, 1.0), "face": (0.0, 0.52, 1.0),
         "edge": (1.0, 0.0, 0.48)}[where]
    return tuple(a * (m - 1) * h for a, m, h in zip(f, n, H))


@pytest.mark.parametrize("n", [(3, 3, 3), (7, 16, 8), (12, 17, 9), (9, 15, 7), (23, 33, 25), (33, 48, 40), (61, 20, 31)])
@pytest.mark.parametrize("where", ["inside", "corner", "end", "face", "edge"])
def test_matches_slabs_and_oracle(fk, n, where):
    vel = _cells(n, sum(n))
    src = _src(n, where)
    for nsweep, eps in ((2, min(3.0, min(n) - 1)), (0, 0.0), (1, float(min(n)))):
        a = _solve(fk, n, vel, src, TILES, 4, nsweep, eps)
        assert np.array_equal(a, _solve(fk, n, vel, src, SLABS, 4, nsweep, eps)), (nsweep, eps)
        d = _solve(fk, n, vel, src, TILES, 8, nsweep, eps)
        si, sa = O.source_snap(True, n, (0, 0, 0), H, src)
        ref, _ = O.solve3d(n, H, 1.0 / vel.ravel(), si, sa, eps, nsweep)
        assert np.max(np.abs(d - ref)) <= 1e-12 * np.max(ref), (nsweep, eps)


def test_precision_change_keeps_the_solver(fk):
    """The edge words are sized by the precision: a change between solves."""
    n = (20, 40, 30)
    vel = layered_grf_cells(*n, seed=1, min_cells=2)
    src = _src(n, "inside")
    want = {p: _solve(fk, n, vel, src, TILES, p) for p in (4, 8)}
    s = fk.fteik3d()
    s.initialize(n[1], n[2], n[0], H[1], H[2], H[0], nsweep=2, eps=5.0, precision=4)
    s.setCellSlownessNatural(vel)
    s.setSources(src[1], src[2], src[0])
    import ctypes
    ierr = ctypes.c_int(1)
    for p in (4, 8, 4, 8):
        fk.lib().fteik_b200_solver3d_setPrecision(p, ctypes.byref(ierr))
        s.solveSourceLSM(1)
        assert np.array_equal(s.getTravelTimeField(), want[p])
    s.free()


@pytest.mark.parametrize("converge", [False, True])
def test_several_launches_match_slabs(fk, converge, tmp_path, monkeypatch):
    """A work list whose tiles pass the chip's: the cached choice makes the
    batch take the tiles, two grids, several sources each."""
    grids = [(60, 96, 90) + H, (33, 50, 41) + H]
    rng = np.random.default_rng(3)
    vels = [layered_grf_cells(*g[:3], seed=i, min_cells=2) for i, g in enumerate(grids)]
    srcs = [tuple(rng.uniform(0, 1, 5) * (m - 1) * h for m, h in zip(g[:3], H)) for g in grids]
    kw = dict(convTol=0.0, maxPass=20) if converge else dict(nsweep=2)
    out = []
    for tiles in (False, True):
        monkeypatch.setenv("FTEIK_B200_TUNE_CACHE", str(tmp_path / "t"))
        old = fk.set_slab_config(*(TILES if tiles else SLABS))
        try:
            b = fk.Batch3D(grids, eps=5.0, precision=4, **kw)
            for i in range(len(grids)):
                b.setVelocityModel(i + 1, vels[i])
                b.setSources(i + 1, *srcs[i])
            if tiles:
                b.solve()         # writes the work list's key, whatever it chose
                line = (tmp_path / "t").read_text().split("\n")[0].rsplit(" ", 1)[0]
                b.finalize()
                (tmp_path / "t").write_text(line + " 1\n")
                # a process that has not tuned this work list reads the file
                import subprocess
                import sys
                code = ("import sys, numpy as np; sys.path[:0] = %r; import fteik_b200 as fk\n"
                        "z = np.load(%r)\n"
                        "b = fk.Batch3D(%r, eps=5.0, precision=4, **%r)\n"
                        "for i in range(2):\n"
                        "    b.setVelocityModel(i + 1, z['v%%d' %% i]); b.setSources(i + 1, *z['s%%d' %% i])\n"
                        "b.solve(); b.solve()\n"
                        "assert b.slabConfig()['tune_runs'] == 0\n"
                        "np.savez(%r, *[b.fields32(i + 1) for i in range(2)])\n"
                        % ([p for p in sys.path if p], str(tmp_path / "in.npz"), grids, kw, str(tmp_path / "out.npz")))
                np.savez(tmp_path / "in.npz", v0=vels[0], v1=vels[1], s0=np.array(srcs[0]), s1=np.array(srcs[1]))
                subprocess.run([sys.executable, "-c", code], check=True, timeout=120)
                z = np.load(tmp_path / "out.npz")
                out.append([z["arr_0"], z["arr_1"]])
            else:
                b.solve()
                out.append([b.fields32(i + 1).copy() for i in range(len(grids))])
                b.finalize()
        finally:
            fk.set_slab_config(*old)
    for a, c in zip(*out):
        assert np.array_equal(a, c)
