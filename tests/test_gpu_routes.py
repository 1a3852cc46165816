"""Calls around the routes by size: FP64 solves on the slabs against the oracle, FP64
batches whose tiles take several launches, observations changed between calls (only
the changed ones are uploaded), and the allocation-free search at sizes that take the
block kernels, on a stream of the caller's and replayed from a captured graph."""
import ctypes
import subprocess
import sys

import numpy as np
import pytest

import oracle_lib as O
from models import layered_grf_cells, station_tables, synthetic_events
from test_gpu_tiles import H, SLABS, TILES, _cells, _solve, _src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(7, 16, 8), (33, 48, 40), (61, 20, 31), (40, 70, 64)])
@pytest.mark.parametrize("where", ["inside", "corner"])
def test_fp64_slabs_match_oracle(fk, n, where):
    vel, src = _cells(n, sum(n)), _src(n, where)
    got = _solve(fk, n, vel, src, SLABS, 8, 2, 3.0)
    si, sa = O.source_snap(True, n, (0, 0, 0), H, src)
    ref, _ = O.solve3d(n, H, 1.0 / vel.ravel(), si, sa, 3.0, 2)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(ref)


def test_fp64_tiles_in_several_launches(fk, tmp_path, monkeypatch):
    """148 FP64 tiles a launch, 77 a source: the cache's choice makes five sources
    take five launches; the same bits as the slabs'."""
    n = (40, 97, 83)
    rng = np.random.default_rng(4)
    vel, src = layered_grf_cells(*n, seed=3, min_cells=2), [rng.uniform(0, 1, 5) * (m - 1) * h for m, h in zip(n, H)]
    monkeypatch.setenv("FTEIK_B200_TUNE_CACHE", str(tmp_path / "t"))

    def batch(cfg):
        old = fk.set_slab_config(*cfg)
        try:
            b = fk.Batch3D([n + H], nsweep=2, eps=5.0, precision=8)
            b.setVelocityModel(1, vel)
            b.setSources(1, *src)
            b.solve()
            out = [b.field(1, k + 1) for k in range(5)]
            b.finalize()
        finally:
            fk.set_slab_config(*old)
        return out
    want = batch(SLABS)
    batch(TILES)                          # writes the work list's key
    line = (tmp_path / "t").read_text().split("\n")[0].rsplit(" ", 1)[0]
    (tmp_path / "t").write_text(line + " 1\n")
    np.savez(tmp_path / "in.npz", vel=vel, src=np.array(src))
    code = ("import sys, numpy as np; sys.path[:0] = %r; import fteik_b200 as fk\n"
            "z = np.load(%r)\n"
            "b = fk.Batch3D([%r], nsweep=2, eps=5.0, precision=8)\n"
            "b.setVelocityModel(1, z['vel']); b.setSources(1, *z['src'])\n"
            "b.solve(); b.solve()\n"
            "assert b.slabConfig()['tune_runs'] == 0 and b.kernelTimes()[0] < 0.1\n"     # no initialisation kernel: tiles
            "np.save(%r, np.array([b.field(1, k + 1) for k in range(5)]))\n"
            % ([p for p in sys.path if p], str(tmp_path / "in.npz"), n + H, str(tmp_path / "out.npy")))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=120)
    for a, c in zip(want, np.load(tmp_path / "out.npy")):
        assert np.array_equal(a, c)


@pytest.mark.parametrize("method,norm", [(0, 2), (0, 1), (1, 2)])
def test_changed_observations_reach_the_search(fk, method, norm):
    ntf, nev = 24, 40
    tables = station_tables(20, 20, 20, 100.0, ntf, seed=6)
    ngrd = tables.shape[1]
    _, first = synthetic_events(tables, nev, seed=1)
    _, later = synthetic_events(tables, nev, seed=2)

    def locator(picks):
        loc = fk.Locator(nev, ntf, ngrd)
        for k in range(ntf):
            loc.setTravelTimeField32f(k + 1, tables[k])
        loc.setMethod(method)
        loc.setNorm(norm)
        for e in range(nev):
            put(loc, picks, e)
        return loc

    def put(loc, picks, e):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], np.full(ntf, 0.5))

    everything = np.arange(1, nev + 1)
    want = []
    for picks in (first, later):
        loc = locator(picks)
        want.append([np.array(v) for v in loc.locateEvents(everything)])
        loc.finalize()
    loc = locator(first)
    now = np.zeros(nev, dtype=int)
    for step in ([], [17], [3, 21, 20], [0], [nev - 1], [5, 38], [], list(range(nev))):
        for e in step:
            put(loc, later, e)
            now[e] = 1
        if len(step) == 1:                # the changed event alone first
            one = loc.locateEvent(step[0] + 1)
            assert one[0] == want[1][0][step[0]]
        got = loc.locateEvents(everything)
        for k in range(3):
            assert np.array_equal(np.array(got[k]), np.where(now, want[1][k], want[0][k])), step
    loc.finalize()


def test_both_copies_of_the_observations(fk):
    """FP32 and FP64 copies are uploaded by different searches, each with its own range."""
    ntf, nev = 24, 30
    tables = station_tables(20, 20, 20, 100.0, ntf, seed=7)
    sets = [synthetic_events(tables, nev, seed=s)[1] for s in (3, 4)]
    loc = fk.Locator(nev, ntf, tables.shape[1])
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    ev = np.arange(1, nev + 1)

    def put(picks, events):
        for e in events:
            loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], np.ones(ntf))

    def both():
        out = []
        for m in (0, 1):
            loc.setMethod(m)
            out.append(np.array(loc.locateEvents(ev)[0]))
        return out
    put(sets[0], range(nev))
    a = both()
    put(sets[1], range(nev))
    b = both()
    put(sets[0], [4, 5])
    loc.setMethod(0)
    loc.locateEvents(ev)                  # FP32 up to date, FP64 not
    put(sets[0], [25])
    c = both()
    for k in range(2):
        assert np.array_equal(c[k], np.where(np.isin(np.arange(nev), [4, 5, 25]), a[k], b[k]))
    loc.finalize()


@pytest.mark.parametrize("ntf,ngrd,nev", [(20, (1 << 18) + 3, 192), (40, (1 << 18) + 1025, 200), (56, (1 << 19) + 5, 193)])
def test_noalloc_at_block_sizes(fk, ntf, ngrd, nev):
    import torch
    tables = np.ascontiguousarray(station_tables(64, 64, ngrd // 4096 + 1, 50.0, ntf, seed=ntf)[:, :ngrd])
    _, picks = synthetic_events(tables, nev, seed=ntf)
    rng = np.random.default_rng(ntf)
    wts = rng.choice([1.0, 0.75, 0.5], picks.shape)
    wts[rng.random(picks.shape) < 0.1] = 0.0
    wts[:, 0] = 1.0
    loc = fk.Locator(nev, ntf, ngrd)
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, tables[k])
    for e in range(nev):
        loc.setObservation(e + 1, np.arange(1, ntf + 1), picks[e], wts[e])
    want = [np.array(v) for v in loc.locateEvents(np.arange(1, nev + 1))]
    loc.finalize()
    tep = picks.max(axis=1)
    obs = np.where(wts > 0, picks - tep[:, None], 0.0).astype(np.float32)
    d = [torch.from_numpy(v).cuda() for v in (tables, obs, wts.astype(np.float32))]
    out = [torch.zeros(nev, dtype=t, device="cuda") for t in (torch.int32, torch.float32, torch.float32)]
    side = torch.cuda.Stream()

    def call():
        ierr = ctypes.c_int(1)
        p = [ctypes.c_void_p(v.data_ptr()) for v in d + out]
        fk.lib().fteik_b200_locate_l2_noalloc(ngrd, ngrd, ntf, p[0], nev, p[1], p[2], p[3], p[4], p[5],
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(ierr))
        assert ierr.value == 0

    def check():
        torch.cuda.synchronize()
        assert np.array_equal(out[0].cpu().numpy() + 1, want[0])
        assert np.array_equal(out[1].cpu().numpy().astype(np.float64) + tep, want[1])
        assert np.array_equal(out[2].cpu().numpy().astype(np.float64), want[2])
        for v in out:
            v.zero_()
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        call()
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call()
    for _ in range(2):
        graph.replay()
        check()
