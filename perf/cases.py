"""The calls a user of this framework spends time in, as measurable cases.

Travel times, 2D and 3D (FP64 drop-in, FP32 single source, FP32 tables of
many sources on one or several grids), grid-search location (one event, a
batch with graded and skipped picks, the L1 norm, the tensor-core search,
the surrogate-pruned search) and the surrogate network (forward, gradient).

The library keeps one instance of each object per process (one 2D and one
3D solver, one batch, one locator, one network), so a case's object is
opened once, when its sizes come up, and stays; a state holds the inputs of
one pass, and a pass gives them to the library and takes the results back.
Velocity models are four layers or a linear gradient, times (1 + 5 % Gaussian
random field); tables for the locator are the exact times of the linear
gradient v = 3000 + 0.5 z (an input of the search: any solver may have made
them).
"""
import math

import numpy as np
import torch

import fteik_b200 as fk

V0, GRAD = 3000.0, 0.5
HUGE = 99999.0
EPS = 5.0
SLOTS = 4               # event ranges of a locator, used in turn by the states
WIDTH, DEPTH = 256, 5   # the surrogate network


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # the plain 2D call: one model, one source, the field back (FP64)
        dict(name="field2d_201", kind="field2d", nz=201, nx=201, h=10.0, nsweep=2),
        # 2D refraction / crosswell forward modelling: every shot to every receiver in one call
        dict(name="times2d_256src", kind="times2d", nz=151, nx=301, h=10.0, nsweep=2, nsrc=256, nrec=96),
        # the reference's own 3D use, in its precision, on a small odd grid
        dict(name="field3d_f64_small", kind="field3d", nz=41, nx=53, ny=47, h=100.0, nsweep=2, precision=8),
        # one source on a mid-size 3D model, iterated until nothing changes (FP32)
        dict(name="field3d_128_converged", kind="tables3d", grids="128x128x128", h=25.0, nsrc=1, converge=True, layers=True),
        # a local network's tables on one ragged grid, brought to the host
        dict(name="tables3d_16src", kind="tables3d", grids="61x97x83", h=200.0, nsrc=16, converge=False, layers=True),
        # many sources on grids of uneven size in one solve, times at the receivers (tomography's forward step)
        dict(name="times3d_64src_4grids", kind="times3d", grids="64x96x96,80x128x128,96x160x160,100x200x120", h=50.0,
             nsrc=64, nrec=400, layers=False),
        # an event just picked: observations in, hypocentre out (quality weights, some picks missing)
        dict(name="locate_one_event", kind="locate", method=0, norm=2, nz=80, nx=128, ny=128, h=50.0, ntf=48, nev=1,
             skipped=0.1, graded=True),
        # relocation of a catalogue with the reference's arithmetic
        dict(name="locate_exact_512", kind="locate", method=0, norm=2, nz=96, nx=160, ny=160, h=50.0, ntf=64, nev=512,
             skipped=0.1, graded=True),
        # the same with the outlier-robust norm
        dict(name="locate_l1_128", kind="locate", method=0, norm=1, nz=96, nx=160, ny=160, h=50.0, ntf=64, nev=128,
             skipped=0.05, graded=False),
        # a synthetic catalogue: every station, one weight
        dict(name="locate_tensor_10000", kind="locate", method=1, norm=2, nz=96, nx=160, ny=160, h=50.0, ntf=64, nev=10000,
             skipped=0.0, graded=False),
        dict(name="locate_pruned_10000", kind="locate", method=2, norm=2, nz=96, nx=160, ny=160, h=50.0, ntf=64, nev=10000,
             skipped=0.0, graded=False),
        # one training step's gradient on host rows
        dict(name="surrogate_grad_16384", kind="mlp", rows=16384, backward=True),
    ]


def _logi(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field2d", "times2d", "field3d", "tables3d", "times3d", "locate", "locate", "locate", "mlp"])
    if kind in ("field2d", "times2d"):
        c = dict(kind=kind, nz=_logi(rng, 41, 520), nx=_logi(rng, 41, 520), h=rng.choice([5.0, 10.0, 25.0]),
                 nsweep=rng.choice([1, 2, 2, 3]))
        if kind == "times2d":
            c.update(nsrc=_logi(rng, 4, 256), nrec=rng.randint(8, 200))
        return c
    if kind == "field3d":
        return dict(kind=kind, nz=_logi(rng, 17, 90), nx=_logi(rng, 17, 90), ny=_logi(rng, 17, 90),
                    h=rng.choice([50.0, 100.0]), nsweep=rng.choice([1, 2, 2, 3]), precision=rng.choice([4, 8]))
    if kind == "tables3d":
        converge = rng.random() < 0.3
        hi = 128 if converge else 110
        g = "x".join(str(_logi(rng, 33, hi)) for _ in range(3))
        return dict(kind=kind, grids=g, h=rng.choice([25.0, 100.0, 200.0]), nsrc=1 if converge else _logi(rng, 2, 32),
                    converge=converge, layers=rng.random() < 0.5)
    if kind == "times3d":
        g = ",".join("x".join(str(_logi(rng, 48, 128)) for _ in range(3)) for _ in range(rng.randint(1, 4)))
        return dict(kind=kind, grids=g, h=rng.choice([50.0, 100.0]), nsrc=_logi(rng, 8, 64), nrec=_logi(rng, 16, 400),
                    layers=rng.random() < 0.5)
    if kind == "mlp":
        return dict(kind=kind, rows=_logi(rng, 500, 65536), backward=rng.random() < 0.6)
    method, norm = rng.choice([(0, 2), (0, 2), (0, 1), (1, 2), (2, 2)])
    c = dict(kind=kind, method=method, norm=norm, nz=_logi(rng, 33, 96), nx=_logi(rng, 48, 160), ny=_logi(rng, 48, 160),
             h=rng.choice([50.0, 100.0]), ntf=rng.randint(10, 64))
    if method == 0:
        most = 512 if norm == 2 else 128
        c.update(nev=1 if rng.random() < 0.3 else _logi(rng, 4, most), skipped=rng.choice([0.0, 0.05, 0.1]),
                 graded=norm == 2 and rng.random() < 0.7)
    else:
        c.update(ntf=rng.randint(24, 64), nev=_logi(rng, 300, 10000), skipped=0.0, graded=False)
    return c


def _grids(case):
    return [tuple(int(v) for v in g.split("x")) for g in case["grids"].split(",")]


def work(case):
    """Bytes: each input read once, each output written once.  Flops: the
    node updates' stencils (about 25 flops in 2D, 90 in 3D; the sweeps of
    the initialisation as one more pass; a converged solve at least one pass
    more than two), the misfits' terms, the network's products."""
    kind = case["kind"]
    if kind in ("field2d", "times2d"):
        n, ns = case["nz"] * case["nx"], case.get("nsrc", 1)
        out = n if kind == "field2d" else ns * case["nrec"]
        return {"bytes": 8 * (n + out), "flops": 25 * n * ns * 4 * (case["nsweep"] + 1)}
    if kind == "field3d":
        n = case["nz"] * case["nx"] * case["ny"]
        return {"bytes": 16 * n, "flops": 90 * n * 8 * (case["nsweep"] + 1)}
    if kind in ("tables3d", "times3d"):
        n, ns = sum(a * b * c for a, b, c in _grids(case)), case["nsrc"]
        out = 4 * n * ns if kind == "tables3d" else 8 * ns * case["nrec"] * len(_grids(case))
        return {"bytes": 8 * n + out, "flops": 90 * n * ns * 8 * (4 if case.get("converge") else 3)}
    if kind == "mlp":
        f = 2 * case["rows"] * (6 * WIDTH + (DEPTH - 1) * WIDTH * WIDTH + WIDTH)
        return {"bytes": 28 * case["rows"] + 4 * _nweights() * (2 if case["backward"] else 1), "flops": f * (3 if case["backward"] else 1)}
    n, ntf, nev = case["nz"] * case["nx"] * case["ny"], case["ntf"], case["nev"]
    if case["method"] == 2:
        return {"bytes": 4 * ntf * min(n, 512 * nev) + 8 * nev * ntf + 20 * nev,
                "flops": 2 * ntf * nev * (n // 64) + 5 * ntf * nev * 512}
    per = 2 if case["method"] == 1 or case["norm"] == 1 else 5
    return {"bytes": 4 * ntf * n + 8 * nev * ntf + 20 * nev, "flops": per * ntf * nev * n}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _smooth(shape, corr, seed):
    """Unit-variance Gaussian random field, correlation of corr cells."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    k2 = 0
    for d, n in enumerate(shape):
        k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) ** 2
        k2 = k2 + k.view([-1 if e == d else 1 for e in range(len(shape))])
    f = torch.fft.ifftn(torch.fft.fftn(w) * torch.exp(-0.5 * k2 * (2 * math.pi * corr) ** 2)).real
    f = (f - f.mean()) / f.std()
    return f.clamp(-3, 3)


def _velocity(shape, h, seed, layers):
    """Cell velocities, z last (fastest)."""
    nzc = shape[-1]
    if layers:
        edges = np.sort(np.random.default_rng(seed).uniform(0.1, 0.9, 3)) * nzc
        vz = 3000.0 + 1000.0 * np.searchsorted(edges, np.arange(nzc) + 0.5)
    else:
        vz = V0 + GRAD * (np.arange(nzc) + 0.5) * h
    v = torch.tensor(vz, device="cuda", dtype=torch.float64) * (1.0 + 0.05 * _smooth(shape, 10.0, seed))
    return v.contiguous()


def _pinned(t):
    """A host copy in page-locked memory, as a program that feeds a GPU keeps its buffers."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def _sources(rng, n, n3, h, surface):
    z = np.zeros(n) if surface else rng.uniform(0.05, 0.95, n) * (n3[0] - 1) * h
    return (z,) + tuple(rng.uniform(0.02, 0.98, n) * (m - 1) * h for m in n3[1:])


_open = {"key": None, "obj": None, "slot": 0}


def _object(key, make):
    """The library's object of these sizes (one at a time in a process)."""
    if _open["key"] != key:
        if _open["obj"] is not None:
            for o in _open["obj"] if isinstance(_open["obj"], tuple) else (_open["obj"],):
                (o.finalize if hasattr(o, "finalize") else o.free)()
        _open.update(key=None, obj=None, slot=0)
        _open.update(key=key, obj=make())
    return _open["obj"]


def _stations(case):
    n3 = (case["nz"], case["nx"], case["ny"])
    rng = np.random.default_rng([n3[0], n3[1], n3[2], case["ntf"]])
    return np.zeros(case["ntf"]), *(rng.uniform(0, (m - 1) * case["h"], case["ntf"]) for m in n3[1:])


def _gradient_times(z, r2, zs):
    """Time from (zs) to (z) at squared distance r2 in v = V0 + GRAD z."""
    lib = torch if isinstance(r2, torch.Tensor) else np
    return lib.arccosh(1.0 + 0.5 * GRAD * GRAD * r2 / ((V0 + GRAD * z) * (V0 + GRAD * zs))) / GRAD


def _table(case, k):
    """FP32 travel times of station k at every node, z fastest (on the GPU)."""
    zs, xs, ys = (s[k] for s in _stations(case))
    z, x, y = (torch.arange(n, device="cuda", dtype=torch.float64) * case["h"] for n in (case["nz"], case["nx"], case["ny"]))
    r2 = (y[:, None, None] - ys) ** 2 + (x[None, :, None] - xs) ** 2 + (z[None, None, :] - zs) ** 2
    return _gradient_times(z[None, None, :], r2, zs).float().reshape(-1)


def _picks(case, seed):
    """Picks and weights [nev][ntf]: exact times of uniform hypocentres + N(0, 0.02 s), 5 % outliers of up to 1 s."""
    rng = np.random.default_rng([7, seed])
    nev, ntf = case["nev"], case["ntf"]
    hz, hx, hy = (rng.uniform(0, (n - 1) * case["h"], (nev, 1)) for n in (case["nz"], case["nx"], case["ny"]))
    zs, xs, ys = _stations(case)
    t = _gradient_times(hz, (hz - zs) ** 2 + (hx - xs) ** 2 + (hy - ys) ** 2, zs) + rng.uniform(0, 60, (nev, 1))
    t = t + np.where(rng.random(t.shape) < 0.05, rng.uniform(-1, 1, t.shape), rng.normal(0, 0.02, t.shape))
    w = rng.choice([1.0, 0.75, 0.5, 0.25], t.shape) if case["graded"] else np.ones(t.shape)
    w[rng.random(t.shape) < case["skipped"]] = 0.0
    w[:, 0] = 1.0
    return t, w


def _locator(case):
    ntf, ngrd = case["ntf"], case["nz"] * case["nx"] * case["ny"]
    loc = fk.Locator(SLOTS * case["nev"], ntf, ngrd)
    for k in range(ntf):
        loc.setTravelTimeField32f(k + 1, _table(case, k).cpu().numpy())
    loc.setNorm(case["norm"])
    if case["method"] < 2:
        loc.setMethod(case["method"])
        return loc
    loc.setGeometry(case["nz"], case["nx"], case["ny"], case["h"], case["h"], case["h"], *_stations(case))
    net = fk.MLP(WIDTH, DEPTH, seed=7)
    loc.trainSurrogate(nsamples=2_000_000, steps=375, batch=65536, lr=4e-3, vref=V0, seed=7)
    loc.buildSurrogate((4, 4, 4))
    loc.setMethod(2)
    return loc, net


def _nweights():
    return 6 * WIDTH + WIDTH + (DEPTH - 1) * (WIDTH * WIDTH + WIDTH) + WIDTH + 1


def _network(seed):
    """Weights as a network in training has them, row-major [out][in] then bias per layer."""
    rng = np.random.default_rng([3, seed])
    dims = [6] + [WIDTH] * DEPTH + [1]
    parts = []
    for i, o in zip(dims, dims[1:]):
        parts += [rng.normal(0, math.sqrt(1.5 / i), i * o), rng.normal(0, 0.05, o)]
    return np.concatenate(parts).astype(np.float32)


def _models(case, seed):
    return [_velocity((ny - 1, nx - 1, nz - 1), case["h"], seed * 16 + i, case["layers"])
            for i, (nz, nx, ny) in enumerate(_grids(case))]


def _inputs(case, seed):
    """Everything of a pass that the seed decides, as exact() needs it too."""
    kind = case["kind"]
    rng = np.random.default_rng([11, seed])
    if kind in ("field2d", "times2d"):
        n2 = (case["nz"], case["nx"])
        vel = _velocity((n2[1] - 1, n2[0] - 1), case["h"], seed, True)
        zs, xs = _sources(rng, case.get("nsrc", 1), n2, case["h"], kind == "times2d")
        s = dict(vel=vel, src=(zs, xs))
        if kind == "times2d":
            s["rec"] = (np.zeros(case["nrec"]), rng.uniform(0, (n2[1] - 1) * case["h"], case["nrec"]))
        return s
    if kind == "field3d":
        n3 = (case["nz"], case["nx"], case["ny"])
        return dict(vel=_velocity((n3[2] - 1, n3[1] - 1, n3[0] - 1), case["h"], seed, True),
                    src=_sources(rng, 1, n3, case["h"], False))
    if kind in ("tables3d", "times3d"):
        gr = _grids(case)
        s = dict(vel=_models(case, seed), src=[_sources(rng, case["nsrc"], g, case["h"], case["nsrc"] > 1) for g in gr])
        if kind == "times3d":
            s["rec"] = [tuple(rng.uniform(0, (m - 1) * case["h"], case["nrec"]) for m in g) for g in gr]
        return s
    if kind == "mlp":
        x = rng.uniform(-1, 1, (case["rows"], 6)).astype(np.float32)
        return dict(w=_network(seed), x=x, y=rng.uniform(0.6, 1.1, case["rows"]).astype(np.float32))
    t, w = _picks(case, seed)
    return dict(picks=t, w=w)


def prepare(case, seed):
    kind, h = case["kind"], case.get("h")
    s = _inputs(case, seed)
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    s["case"] = case

    if kind in ("field2d", "times2d"):
        def make():
            o = fk.fteik2d()
            o.initialize(case["nx"], case["nz"], h, h, nsweep=case["nsweep"], eps=EPS)
            return o
        s["obj"] = _object(key, make)
        s["vel"] = _pinned(s["vel"])
    elif kind == "field3d":
        def make():
            o = fk.fteik3d()
            o.initialize(case["nx"], case["ny"], case["nz"], h, h, h, nsweep=case["nsweep"], eps=EPS,
                         precision=case["precision"])
            return o
        s["obj"] = _object(key, make)
        s["vel"] = _pinned(s["vel"])
    elif kind in ("tables3d", "times3d"):
        gr = _grids(case)

        def make():
            conv = dict(convTol=0.0, maxPass=30) if case.get("converge") else {}
            return fk.Batch3D([(nz, nx, ny, h, h, h) for nz, nx, ny in gr], nsweep=2, eps=EPS, precision=4, **conv)
        s["obj"] = _object(key, make)
        s["vel"] = [_pinned(v) for v in s["vel"]]
        if kind == "tables3d":
            n = case["nsrc"] * gr[0][0] * gr[0][1] * gr[0][2]
            s["out"] = torch.empty(n, dtype=torch.float32, pin_memory=True).numpy()
    elif kind == "mlp":
        s["obj"] = _object("mlp", lambda: fk.MLP(WIDTH, DEPTH, seed=7))
    else:
        loc = _object(key, lambda: _locator(case))
        s["obj"] = loc[0] if isinstance(loc, tuple) else loc
        nev, ntf = case["nev"], case["ntf"]
        s["ev"] = np.arange(1, nev + 1, dtype=np.int32) + nev * (_open["slot"] % SLOTS)
        _open["slot"] += 1
        s["obs2tf"] = np.arange(1, ntf + 1, dtype=np.int32)
        if nev > 1:      # a catalogue's picks are on file before it is relocated
            for e, p, w in zip(s["ev"], s["picks"], s["w"]):
                s["obj"].setObservation(e, s["obs2tf"], p, w)
    return s


def run(state):
    case, o = state["case"], state["obj"]
    kind = case["kind"]
    if kind in ("field2d", "times2d"):
        o.setCellVelocityNatural(state["vel"])
        zs, xs = state["src"]
        o.setSources(xs, zs)
        if kind == "field2d":
            o.solveSourceLSM(1)
            return o.getTravelTimeField()
        o.setReceivers(state["rec"][1], state["rec"][0])
        o.solveLSM()
        return o.getTravelTimes()
    if kind == "field3d":
        o.setCellSlownessNatural(state["vel"])
        zs, xs, ys = state["src"]
        o.setSources(xs, ys, zs)
        o.solveSourceLSM(1)
        return o.getTravelTimeField()
    if kind in ("tables3d", "times3d"):
        for g, (v, src) in enumerate(zip(state["vel"], state["src"]), start=1):
            o.setVelocityModel(g, v)
            o.setSources(g, *src)
            if kind == "times3d":
                o.setReceivers(g, *state["rec"][g - 1])
        o.solve()
        if kind == "tables3d":
            return o.fields32(1, state["out"])
        return [o.travelTimes(g) for g in range(1, len(state["vel"]) + 1)]
    if kind == "mlp":
        o.setWeights(state["w"])
        return o.gradient(state["x"], state["y"]) if case["backward"] else o.forward(state["x"])
    if case["nev"] == 1:
        e = int(state["ev"][0])
        o.setObservation(e, state["obs2tf"], state["picks"][0], state["w"][0])
        return o.locateEvent(e)
    return o.locateEvents(state["ev"])


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------

def _snap(n, h, v):
    """Grid coordinate (1-based) of a source and its cell."""
    a = v / h + 1.0
    a = np.where(np.abs(a - 1.0) < np.finfo(float).eps, a + 1e-4, a)
    a = np.where(a >= n, a - 1e-4, a)
    return a, a.astype(np.int64)


def _levels(shape):
    """Flat indices of the nodes with every coordinate >= 1, by the sum of the coordinates."""
    grids = torch.meshgrid(*[torch.arange(n, device="cuda") for n in shape], indexing="ij")
    inner = torch.stack([g >= 1 for g in grids]).all(0).reshape(-1)
    lev = sum(grids).reshape(-1)
    idx = torch.nonzero(inner)[:, 0]
    order = torch.argsort(lev[idx], stable=True)
    idx = idx[order]
    return torch.split(idx, torch.bincount(lev[idx]).tolist())


def _cells(slow, axis, side):
    """Cell values re-indexed by node: the cell before (side 0) or after (side 1) a node, clamped."""
    n = slow.shape[axis] + 1
    i = torch.arange(n, device="cuda")
    return slow.index_select(axis, (i - 1).clamp(min=0) if side == 0 else i.clamp(max=n - 2))


def _both(slow, axis):
    return torch.minimum(_cells(slow, axis, 0), _cells(slow, axis, 1))


def _plane(ta, tb, s, ca, cb):
    """Plane-wave time of two axes: ta with 1/h^2 of axis a (ca), tb with cb."""
    tab = ta - tb
    return ((tb * cb + ta * ca) + torch.sqrt(4.0 * s * s * (ca + cb) - ca * cb * tab * tab)) / (ca + cb)


class _Sweeps:
    """Level-ordered sweeps of all sources of one grid at once; axes (y, x, z) or (x, z), arrays [nodes, sources]."""

    def __init__(self, vel, h, src):
        self.h, self.slow = h, 1.0 / vel
        self.shape = tuple(n + 1 for n in vel.shape)
        self.dim = len(self.shape)
        self.ns = len(src[0])
        d = dict(device="cuda", dtype=torch.float64)
        snapped = [_snap(n, h, s) for n, s in zip(self.shape, (src[::-1] if self.dim == 2 else (src[2], src[1], src[0])))]
        self.a = [torch.tensor(a, **d) for a, _ in snapped]                    # per axis [ns], 1-based coordinate
        self.i = [torch.tensor(i, device="cuda") for _, i in snapped]          # 1-based cell
        self.szero = self.slow[tuple(i - 1 for i in self.i)]
        self.level = _levels(self.shape)
        stride = [1] * self.dim
        for k in range(self.dim - 2, -1, -1):
            stride[k] = stride[k + 1] * self.shape[k + 1]
        self.stride = stride
        co = torch.meshgrid(*[torch.arange(n, **d) for n in self.shape], indexing="ij")
        self.diff = [((c.reshape(-1, 1) + 1.0) - a) * h for c, a in zip(co, self.a)]
        self.d0 = torch.sqrt(sum(v * v for v in self.diff))
        self.ana = self.szero * self.d0
        self.tt = torch.full((math.prod(self.shape), self.ns), HUGE, **d)
        for m in range(1 << self.dim):
            f = sum((i - 1 + ((m >> k) & 1)) * s for k, (i, s) in enumerate(zip(self.i, stride)))
            self.tt[f, torch.arange(self.ns, device="cuda")] = self.ana[f, torch.arange(self.ns, device="cuda")]

    def flip(self, a, axes):
        return a.reshape(*self.shape, -1).flip(axes).reshape(a.shape[0], -1) if axes else a

    def sweep(self, axes, init):
        """One sweep with the axes in `axes` walked downwards."""
        tt = self.flip(self.tt, axes).contiguous()
        slow = self.slow.flip(axes) if axes else self.slow
        up = [1 if k not in axes else -1 for k in range(self.dim)]
        if self.dim == 2:
            s = [_cells(_both(slow, 0), 1, 0), _cells(_both(slow, 1), 0, 0), _cells(_cells(slow, 0, 0), 1, 0)]
            off = [-self.stride[1], -self.stride[0], -self.stride[1] - self.stride[0]]
        else:
            Y, X, Z = 0, 1, 2
            lo = lambda a, *ax: _cells(lo(a, *ax[1:]), ax[0], 0) if ax else a          # noqa: E731
            mn = lambda a, *ax: _both(mn(a, *ax[1:]), ax[0]) if ax else a              # noqa: E731
            s = [lo(mn(slow, X, Y), Z), lo(mn(slow, Z, Y), X), lo(mn(slow, Z, X), Y), lo(mn(slow, Y), Z, X),
                 lo(mn(slow, X), Z, Y), lo(mn(slow, Z), X, Y), lo(slow, X, Y, Z)]
            z, x, y = self.stride[2], self.stride[1], self.stride[0]
            off = [-z, -x, -y, -z - x, -x - y, -z - y, -z - x - y]
        s = torch.stack([v.reshape(-1) for v in s])
        off = torch.tensor(off + [0], device="cuda")[:, None]
        if init:
            ana, d0 = self.flip(self.ana, axes), self.flip(self.d0, axes)
            diff = [self.flip(v, axes) for v in self.diff]
            lo = [torch.maximum(i - 1, torch.ones_like(i)) if u > 0 else torch.maximum(n - i - 1, torch.ones_like(i))
                  for i, u, n in zip(self.i, up, self.shape)]
        for idx in self.level:
            if not idx.numel():
                continue
            t = tt[idx[None] + off]
            sl = s[:, idx][..., None]
            if not init:
                new = self.plain2(t, sl) if self.dim == 2 else self.plain3(t, sl)
            else:
                co, rest = [], idx
                for st in self.stride:
                    co.append((rest // st)[:, None])
                    rest = rest % st
                inside = torch.ones_like(t[-1], dtype=torch.bool)
                for c, b in zip(co, lo):
                    inside &= c >= b
                if not bool(inside.any()):
                    continue
                tau = t - ana[idx[None] + off]
                r = d0[idx]
                gi = torch.where(r > 0, self.szero / r.clamp(min=1e-300), torch.zeros_like(r))
                tc = [gi * v[idx] * u / self.h for v, u in zip(diff, up)]      # sign * d(tau0)/dx / h per axis
                orig = [(c + 1 if u > 0 else n - c) for c, u, n in zip(co, up, self.shape)]
                new = (self.first2 if self.dim == 2 else self.first3)(t, sl, tau, ana[idx], tc, orig)
                new = torch.where(inside, new, t[-1])
            tt[idx] = torch.minimum(t[-1], new)
        old, self.tt = self.tt, self.flip(tt, axes)
        return float((self.tt - old).abs().max())

    def plain2(self, t, s):
        tv, te, tev, _ = t
        h, c = self.h, 1.0 / (self.h * self.h)
        best = torch.minimum(tv + h * s[0], te + h * s[1])
        d = te - tv
        on = (d < h * s[2]) & (-d < h * s[2])
        return torch.where(on, torch.minimum(best, _plane(tev + d, tev - d, s[2], c, c)), best)

    def first2(self, t, s, tau, t0c, tc, orig):
        tv, te, tev, _ = t
        h, c, s3 = self.h, 1.0 / (self.h * self.h), s[2]
        far = ((orig[0] - self.i[0]).abs() > EPS) | ((orig[1] - self.i[1]).abs() > EPS)
        best = torch.minimum(tv + h * s[0], te + h * s[1])
        huge = torch.full_like(tv, HUGE)
        up = (te >= tev) & (tv >= tev)
        flat = (tv <= te + h * s3) & (te <= tv + h * s3) & up
        lim = h * h * s3 / math.sqrt(2.0 * h * h)
        a = torch.where(flat, _plane(tev + te - tv, tev - te + tv, s3, c, c), huge)
        ex = ~flat & (te - tev <= lim) & (te > tev)
        a = torch.where(ex, te + h * torch.sqrt(s3 * s3 - ((te - tev) / h) ** 2), a)
        ez = ~flat & ~ex & (tv - tev <= lim) & (tv > tev)
        a = torch.where(ez, tv + h * torch.sqrt(s3 * s3 - ((tv - tev) / h) ** 2), a)
        u, e, d = tau[0], tau[1], tau[2]
        ta, tb = d + e - u, d - e + u
        ap = 2.0 * c
        bp = 4.0 * (tc[0] + tc[1]) - 2.0 * (ta * c + tb * c)
        # tc carries the axis sign and 1/h once, as the constant terms want it
        cp = ta * ta * c + tb * tb * c - 4.0 * (tc[0] * ta + tc[1] * tb) + 4.0 * (self.szero ** 2 - s3 * s3)
        dp = bp * bp - 4.0 * ap * cp
        r = 0.5 * (torch.sqrt(dp.clamp(min=0.0)) - bp) / ap + t0c
        ok = (dp >= 0) & (tv < te + h * s3) & (te < tv + h * s3) & up & (r >= tv) & (r >= te)
        return torch.minimum(best, torch.where(far, a, torch.where(ok, r, huge)))

    def cube(self, tv, te, tn, tev, ten, tnv, tnve):
        return (te + 0.5 * (-tn + ten - tv + tev) - tnv + tnve, tv + 0.5 * (-tn + tnv - te + tev) - ten + tnve,
                tn + 0.5 * (-te + ten - tv + tnv) - tev + tnve)

    def volume(self, t, s):
        """3D plane-wave operator, HUGE where it has no solution."""
        c = 1.0 / (self.h * self.h)
        ta, tb, tc = self.cube(*t[:7])
        q = 9.0 * (3.0 * c) * s * s - c * c * ((ta - tb) ** 2 + (tb - tc) ** 2 + (ta - tc) ** 2)
        r = ((ta + tb + tc) * c + torch.sqrt(q.clamp(min=0.0))) / (3.0 * c)
        return torch.where(q >= 0, r, torch.full_like(r, HUGE))

    def plain3(self, t, s):
        tv, te, tn, tev, ten, tnv = t[:6]
        h, c = self.h, 1.0 / (self.h * self.h)
        best = torch.minimum(torch.minimum(tv + h * s[0], te + h * s[1]), tn + h * s[2])
        for a, b, ab, sl in ((te, tv, tev, s[3]), (tv, tn, tnv, s[4]), (te, tn, ten, s[5])):
            d = a - b
            on = (d < h * sl) & (-d < h * sl)
            best = torch.where(on, torch.minimum(best, _plane(ab + d, ab - d, sl, c, c)), best)
        top = torch.maximum(torch.maximum(tv, te), tn)
        return torch.where(best > top, torch.minimum(best, self.volume(t, s[6])), best)

    def first3(self, t, s, tau, t0c, tc, orig):
        tv, te, tn, tev, ten, tnv = t[:6]
        h, c = self.h, 1.0 / (self.h * self.h)
        ty, tx, tz = tc
        huge = torch.full_like(tv, HUGE)
        best = torch.minimum(torch.minimum(tv + h * s[0], te + h * s[1]), tn + h * s[2])
        low = torch.minimum(torch.minimum(tv, te), tn)
        top = torch.maximum(torch.maximum(tv, te), tn)
        cart = low > EPS * h * self.szero
        uv, ue, un, uev, uen, unv, unve = tau[:7]
        # (time a, b, ab; tau a, b, ab; slowness; gradients a, b, other; the axis the source plane lies on)
        for a, b, ab, qa, qb, qab, sl, ga, gb, go, k in (
                (te, tv, tev, ue, uv, uev, s[3], tx, tz, ty, 0), (tv, tn, tnv, uv, un, unv, s[4], tz, ty, tx, 1),
                (te, tn, ten, ue, un, uen, s[5], tx, ty, tz, 2)):
            on = (a < b + h * sl) & (b < a + h * sl)
            flat = cart | (orig[k] != self.i[k])
            p = _plane(ab + a - b, ab - a + b, sl, c, c)
            ta, tb = qab + qa - qb, qab - qa + qb
            ap = 2.0 * c
            bp = 4.0 * (ga + gb) - 2.0 * (ta + tb) * c
            cp = (ta * ta + tb * tb) * c - 4.0 * (ga * ta + gb * tb) + 4.0 * (self.szero ** 2 - sl * sl + (go * h) ** 2)
            dp = bp * bp - 4.0 * ap * cp
            r = (torch.sqrt(dp.clamp(min=0.0)) - bp) / (2.0 * ap) + t0c
            r = torch.where((dp >= 0) & (r >= a) & (r >= b), r, huge)
            best = torch.where(on, torch.minimum(best, torch.where(flat, p, r)), best)
        vol = self.volume(t, s[6])
        qa, qb, qc = self.cube(*tau[:7])
        ap = 3.0 * c
        bp = 6.0 * (tz + ty + tx) - 2.0 * (qa + qb + qc) * c
        cp = (qa * qa + qb * qb + qc * qc) * c - 6.0 * (tx * qa + tz * qb + ty * qc) + 9.0 * (self.szero ** 2 - s[6] ** 2)
        dp = bp * bp - 4.0 * ap * cp
        r = (torch.sqrt(dp.clamp(min=0.0)) - bp) / (2.0 * ap) + t0c
        r = torch.where((dp >= 0) & (r >= te) & (r >= tn) & (r >= tv), r, huge)
        return torch.where(best > top, torch.minimum(best, torch.where(cart, vol, r)), best)

    def solve(self, nsweep, converge=False):
        if self.dim == 2:      # order of the sweeps: x down on the even ones, then z down
            order = [(), (0,), (1,), (0, 1)]
        else:                  # s: z down for s >= 5, x on even s, y on 3, 4, 7, 8
            order = [tuple(k for k, on in ((0, s // 2 % 2), (1, s % 2), (2, s >= 4)) if on) for s in range(8)]
        for axes in order:
            self.sweep(axes, True)
        for _ in range(30 if converge else nsweep):
            if max([self.sweep(axes, False) for axes in order]) <= 0.0 and converge:
                break
        return self.tt

    def at(self, rec):
        """Multilinear interpolation at the receivers, [nrec, ns]; rec per axis in the order of src."""
        pts = rec[::-1] if self.dim == 2 else (rec[2], rec[1], rec[0])
        out = 0
        cell, frac = [], []
        for p, n in zip(pts, self.shape):
            p = torch.tensor(p, device="cuda", dtype=torch.float64) / self.h
            i = p.floor().clamp(0, n - 2)
            cell.append(i.long())
            frac.append(p - i)
        for m in range(1 << self.dim):
            w, f = 1.0, 0
            for k in range(self.dim):
                bit = (m >> k) & 1
                w = w * (frac[k] if bit else 1.0 - frac[k])
                f = f + (cell[k] + bit) * self.stride[k]
            out = out + w[:, None] * self.tt[f]
        return out


def _search(case, picks, w):
    """Exhaustive search in 64 bits: (None, t0, misfit) per event."""
    tables = torch.stack([_table(case, k) for k in range(case["ntf"])])
    nev, ngrd = case["nev"], tables.shape[1]
    top = torch.tensor(picks.max(1), device="cuda")
    o = torch.tensor(picks, device="cuda") - top[:, None]
    w = torch.tensor(w, device="cuda")
    best = torch.full((nev,), math.inf, device="cuda", dtype=torch.float64)
    node = torch.zeros(nev, device="cuda", dtype=torch.long)
    if case["norm"] == 2:
        wn, w2 = w / w.sum(1, keepdim=True), w * w
        step = max(256, (1 << 26) // nev)
        for a in range(0, ngrd, step):
            t = tables[:, a:a + step].double()
            t0 = (wn * o).sum(1, keepdim=True) - wn @ t
            # sum w2 (o - t - t0)^2, the cross terms as products
            s1 = (w2 * o).sum(1, keepdim=True) - w2 @ t
            s2 = (w2 * o * o).sum(1, keepdim=True) - 2.0 * (w2 * o) @ t + w2 @ (t * t)
            v, j = (s2 - 2.0 * t0 * s1 + t0 * t0 * w2.sum(1, keepdim=True)).min(1)
            node = torch.where(v < best, j + a, node)
            best = torch.minimum(best, v)
    else:
        # pairs of picks bound the misfit from below: sum |r_i - t| >= |r_i - r_j|
        for e in range(nev):
            used = torch.nonzero(w[e] > 0)[:, 0]
            r = (o[e, used][:, None] - tables[used].double())
            half = len(used) // 2
            bound = (r[:half] - r[half:2 * half]).abs().sum(0)
            def full(q):
                return (q - q.quantile(0.5, 0, keepdim=True)).abs().sum(0)
            upper = full(r[:, bound.argmin().view(1)])
            keep = torch.nonzero(bound <= upper * (1 + 1e-12))[:, 0]
            node[e] = min(((v.min().item(), keep[a + int(v.argmin())].item()) for a in range(0, len(keep), 1 << 16)
                           for v in (full(r[:, keep[a:a + (1 << 16)]]),)))[1]
    r = o - tables[:, node].T.double()
    if case["norm"] == 2:
        t0 = (w * r).sum(1) / w.sum(1)
        obj = 0.5 * ((w * (r - t0[:, None])) ** 2).sum(1)
    else:
        t0 = torch.stack([r[e, w[e] > 0].quantile(0.5) for e in range(nev)])
        obj = (w * (r - t0[:, None]).abs()).sum(1)
    return None, (t0 + top).cpu().numpy(), obj.cpu().numpy()


def _mlp(case, s):
    p = torch.tensor(s["w"], device="cuda", dtype=torch.float64, requires_grad=case["backward"])
    a, at = torch.tensor(s["x"], device="cuda").double(), 0
    dims = [6] + [WIDTH] * DEPTH + [1]
    for k, (i, o) in enumerate(zip(dims, dims[1:])):
        W, b = p[at:at + i * o].view(o, i), p[at + i * o:at + i * o + o]
        at += i * o + o
        a = a @ W.T + b
        a = torch.nn.functional.silu(a) if k < DEPTH else a
    if not case["backward"]:
        return a[:, 0].cpu().numpy()
    loss = ((a[:, 0] - torch.tensor(s["y"], device="cuda").double()) ** 2).mean()
    loss.backward()
    return float(loss), p.grad.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tables3d", "times3d"):
        # level by level with torch: too slow beyond these
        n = sum(a * b * c for a, b, c in _grids(case))
        if n * case["nsrc"] * (8 if case.get("converge") else 3) > 1e8 or len(_grids(case)) > 1:
            return None
    s = _inputs(case, seed)
    if kind == "mlp":
        return _mlp(case, s)
    if kind == "locate":
        got = _search(case, s["picks"], s["w"])
        return (None, float(got[1][0]), float(got[2][0])) if case["nev"] == 1 else got
    if kind in ("field2d", "times2d"):
        f = _Sweeps(s["vel"], case["h"], s["src"])
        f.solve(case["nsweep"])
        return f.tt[:, 0].cpu().numpy() if kind == "field2d" else f.at(s["rec"]).T.contiguous().cpu().numpy()
    if kind == "field3d":
        return _Sweeps(s["vel"], case["h"], s["src"]).solve(case["nsweep"])[:, 0].cpu().numpy()
    f = _Sweeps(s["vel"][0], case["h"], s["src"][0])
    f.solve(2, case.get("converge", False))
    if kind == "tables3d":
        return f.tt.T.contiguous().cpu().numpy().reshape(-1)
    return [f.at(s["rec"][0]).T.contiguous().cpu().numpy()]
