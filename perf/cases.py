"""The work whose time is watched: the calls a program makes of this package, over their range.

A case is a dict of plain values; its "path" says which public entry points it goes through:

  noalloc   capi.advance_noalloc on the caller's own device buffers (real-time loops, plug-in hosts)
  engine    capi.Engine with every snapshot resident in its ring: new seeds on the device, one run, the
            results fetched (how a program uses one field for many seed sets)
  host      TrajectoryIntegrator(settings, loader, TrajectorySet(seeds)).compute(): every snapshot comes
            from host memory through the loader, the records go back to it
  batch     capi.Batch: seed sets of uneven size and lifetime on a 3D and a 2D field, one graph replay
  serve     capi.Server: requests of uneven size, start and length, submitted together

"run" says what is computed: "positions" (final positions and abort codes), "plain" (total curvature, a
temperature volume, the expression sqrt(u*u+v*v)*T, records on the way), "precise" (Kahan positions, float64
time weights, total curvature), "general" (uplift, per-particle constants and a volume that change with time, two
expressions, individual curvature, abort at a path length).  "border" is the border mode (0 Block, 1 LoopX,
3 LoopXY; 2D), "sphere" the 2D fields on a sphere in degrees.

Fields are sums of plane waves with amplitudes ~ |k|^(-5/3), seeds uniform in the lower half of the domain, steps
60 s long with snapshots 600 s apart (1 km, 1 km, 250 m), like the benchmark's configurations; the double gyre
is the 2D analytic field.  All sizes, types and directions that the entry points take may be drawn.
"""
import math

import numpy as np
import torch

import pygranite_b200 as pg
from pygranite_b200 import capi
from pygranite_b200 import workloads

DEVICE = "cuda"
H, SPACING = 60.0, 600.0                 # step and snapshot distance, seconds
PER_WINDOW = 10                          # steps from one snapshot to the next
STORES = {"f32": 0, "bf16": 1, "f16": 2}
EXPRESSION = "sqrt(u*u+v*v)*T"
GENERAL = ("sqrt(u*u+v*v)*T+c", "T-0.5*w+z*0.001")
MODES = 12
BASE = {"path": "engine", "dim": 3, "rk4": 1, "nz": 64, "ny": 192, "nx": 192, "n": 10_000, "steps": 100,
        "store": "f32", "run": "positions", "save": 0, "border": 0, "sphere": 0, "sets": 0}


def case(**kw):
    return dict(BASE, **kw)


def listed():
    return [
        # a control loop that moves a thousand tracers by one snapshot window, on a coarse model grid
        case(name="noalloc small", path="noalloc", nz=16, ny=24, nx=24, n=1000, steps=10),
        # the same call in a plug-in host that owns a large cloud, two windows' worth of steps
        case(name="noalloc large", path="noalloc", n=500_001, steps=20),
        # the 2D double gyre with the defaults of a script: pageable arrays, every step recorded
        case(name="host gyre", path="host", dim=2, rk4=0, nz=1, ny=128, nx=256, n=10_000, steps=1024, save=1,
             run="gyre"),
        # the plain 3D configuration through the loader, page-locked arrays both ways
        case(name="host plain", path="host", n=200_000, steps=100, run="plain", save=10),
        # a few thousand seeds (one station network, one release) on a resident field
        case(name="engine small", n=4097, steps=240, run="plain", save=10),
        # the plain 3D configuration at its particle count
        case(name="engine plain", n=1_000_000, steps=300, run="plain", save=10),
        # final positions only in 16-bit wind storage on the serving grid, ragged count
        case(name="engine bf16", nz=96, ny=512, nx=512, n=777_777, steps=100, store="bf16"),
        # the precision form
        case(name="engine precise", n=250_000, steps=150, run="precise", save=50),
        # every option at once: an ensemble with uplift, constants, volumes, curvature records, length abort
        case(name="engine general", n=65_000, steps=100, run="general", save=5),
        # a global 2D field in degrees, looping in longitude
        case(name="engine 2d sphere", dim=2, nz=1, ny=121, nx=360, n=150_000, steps=200, border=1, sphere=1, save=20),
        # uneven seed sets on two fields as one graph
        case(name="batch", path="batch", n=20_000, steps=600, store="bf16", sets=48),
        # a burst of requests
        case(name="serve", path="serve", n=20_000, steps=400, store="bf16", sets=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["noalloc", "noalloc", "engine", "engine", "engine", "engine", "host", "batch", "serve"])
    dim = rng.choice([2, 3, 3])
    c = dict(path=path, dim=dim, rk4=rng.choice([0, 1, 1, 1]), store=rng.choice(["f32", "f32", "bf16", "f16"]))
    if dim == 3:
        c.update(nz=rng.randint(12, 80), ny=rng.randint(20, 220), nx=rng.randint(20, 220))
    else:
        c.update(nz=1, ny=rng.randint(60, 600), nx=rng.randint(100, 1100))
    if path == "noalloc":
        c.update(store="f32", n=_log(rng, 500, 600_000), steps=_log(rng, 1, 40))
    elif path == "engine":
        run = rng.choice(["positions", "plain", "plain", "precise", "general"])
        if dim == 2 and run != "plain":
            run = "positions"
        most = {"positions": 800_000, "plain": 700_000, "precise": 400_000, "general": 60_000}[run]
        c.update(run=run, n=_log(rng, 1000, most), steps=rng.randint(30, 250))
        c.update(save=0 if run == "positions" and rng.random() < 0.7 else rng.randint(5, 30))
    elif path == "host":
        c.update(run=rng.choice(["positions", "plain"]), n=_log(rng, 1000, 250_000), steps=rng.randint(20, 120))
        c.update(save=rng.choice([0, 5, 10]) if c["run"] == "positions" else 10, store="f32")
    else:
        c.update(dim=3, nz=rng.randint(12, 70), ny=rng.randint(20, 200), nx=rng.randint(20, 200), rk4=1,
                 n=_log(rng, 1000, 30_000), steps=rng.randint(100, 500), sets=rng.randint(3, 20))
    if c["dim"] == 2 and path in ("noalloc", "engine"):
        c.update(border=rng.choice([0, 1, 3]))
    return case(**c)


# ----------------------------------------------------------------- inputs

def _shape(c):
    return (c["nz"], c["ny"], c["nx"]) if c["dim"] == 3 else (c["ny"], c["nx"])


def _cell(c):
    """Grid scale and offset per axis, x first."""
    if c["run"] == "gyre":
        return [2.0 / c["nx"], 1.0 / c["ny"]], [0.0, 0.0]
    if c["sphere"]:
        return [360.0 / c["nx"], 120.0 / c["ny"]], [0.0, -60.0]
    return [1000.0, 1000.0, 250.0][:c["dim"]], [0.0] * c["dim"]


def _radius(c):
    return 6_371_000.0 if c["sphere"] else 0.0


def _step(c):
    """Step and snapshot distance; both exact in binary, so a window holds a whole number of steps."""
    return (1.0 / 128, 1.0) if c["run"] == "gyre" else (H, SPACING)


def _per_window(c):
    h, d = _step(c)
    return int(round(d / h))


def _snapshots(c):
    return -(-c["steps"] // _per_window(c)) + 1


class Field:
    """Snapshots of a sum of plane waves per component, evaluated on the GPU."""

    def __init__(self, c, seed, dim=None, shape=None):
        self.shape = shape or _shape(c)
        self.dim = dim or c["dim"]
        self.gyre = c["run"] == "gyre"
        rng = np.random.default_rng(seed)
        self.seed = seed
        spacing = [250.0, 1000.0, 1000.0][-self.dim:]
        axes = [torch.arange(n, dtype=torch.float64, device=DEVICE) * d for n, d in zip(self.shape, spacing)]
        top, low = 2 * math.pi / 4000.0, 2 * math.pi / max(n * d for n, d in zip(self.shape, spacing))
        self.parts = []
        for k in range(self.dim):
            size = np.exp(rng.uniform(math.log(min(low, top)), math.log(top), MODES))
            way = rng.normal(size=(MODES, self.dim))
            if self.dim == 3:
                way[:, 0] *= 0.25
            vec = size[:, None] * way / np.linalg.norm(way, axis=1, keepdims=True)
            amp = size ** (-5.0 / 3.0)
            amp *= (0.1 if k == 2 else 7.0710678) / math.sqrt(0.5 * float(np.sum(amp * amp)))
            phase, drift = rng.uniform(0, 2 * math.pi, MODES), vec[:, -1] * 5.0 + vec[:, -2] * 3.0
            waves = [torch.exp(1j * torch.outer(torch.as_tensor(vec[:, a], device=DEVICE), axes[a])).to(torch.complex64)
                     for a in range(self.dim)]
            plane = waves[-1] if self.dim == 2 else (waves[1][:, :, None] * waves[2][:, None, :]).reshape(MODES, -1)
            self.parts.append((amp, phase, drift, waves[0], plane))

    def snapshot(self, k):
        """float32 planes (z, y, x) or (y, x) of snapshot k."""
        if self.gyre:
            return self._gyre(k)
        out = []
        for amp, phase, drift, lead, plane in self.parts:
            coef = torch.as_tensor(amp * np.exp(1j * (phase - drift * SPACING * k)), device=DEVICE).to(torch.complex64)
            out.append(((coef[:, None] * lead).T @ plane).real.reshape(self.shape).contiguous())
        return out

    def _gyre(self, k):
        """The double gyre with an amplitude and a phase of this seed, at time k."""
        rng = np.random.default_rng(self.seed)
        a, shift = 0.1 * rng.uniform(0.8, 1.2), rng.uniform(0, 2 * math.pi)
        ny, nx = self.shape
        y, x = torch.meshgrid(torch.arange(ny, dtype=torch.float64, device=DEVICE) / ny,
                              torch.arange(nx, dtype=torch.float64, device=DEVICE) * (2.0 / nx), indexing="ij")
        e = 0.25 * math.sin(2 * math.pi / 10 * k + shift)
        f, slope = e * x * x + (1 - 2 * e) * x, 2 * e * x + 1 - 2 * e
        u = -math.pi * a * torch.sin(math.pi * f) * torch.cos(math.pi * y)
        v = math.pi * a * torch.cos(math.pi * f) * torch.sin(math.pi * y) * slope
        return [u.float().contiguous(), v.float().contiguous()]


def _seeds(c, seed, n=None, dim=None, shape=None):
    dim, shape = dim or c["dim"], shape or _shape(c)
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 7 + 1)
    at = torch.rand((n or c["n"], dim), generator=gen, device=DEVICE, dtype=torch.float64)
    scale, off = _cell(c)
    size = [shape[-1 - d] * scale[d] * (0.5 if d == 2 else 1.0) for d in range(dim)]
    return (at * torch.tensor(size, device=DEVICE) + torch.tensor(off[:dim], device=DEVICE)).float()


def _temperature(c, seed, k=0):
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 31 + k + 5)
    shape = _shape(c)
    z = torch.arange(shape[0], device=DEVICE, dtype=torch.float32).reshape((-1,) + (1,) * (len(shape) - 1)) * 250.0
    return (290.0 - 6.5e-3 * z + 2.0 * torch.randn(shape, generator=gen, device=DEVICE)).contiguous()


def _constant(c, seed, k):
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 37 + k + 11)
    return torch.rand(c["n"], generator=gen, device=DEVICE) * 4.0


def _uplift(c, seed, k):
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 41 + k + 17)
    return torch.randn((c["n"], 3), generator=gen, device=DEVICE) * torch.tensor([2.0, 2.0, 0.5], device=DEVICE)


MAX_LENGTH = 30_000.0


def _reference(c):
    """IntegratorSettings field values, by their names."""
    scale, off = _cell(c)
    h, d = _step(c)
    plain, general = c["run"] == "plain", c["run"] == "general"
    s = dict(Space=0 if c["dim"] == 3 else 1, Integrator=c["rk4"], WindfieldMode=1, DeltaT=h, DataTimeDistance=d,
             GridScale=scale, Offset=off, SaveInterval=c["save"], BorderMode=c["border"], SphereRadius=_radius(c),
             MaximumSimulationTime=h * c["steps"], CurvatureMode=0)
    if c["dim"] == 3 and c["run"] in ("plain", "precise"):
        s.update(CurvatureMode=1)
    if plain:
        s.update(AdditionalVolumeMode=1)
    if general:
        s.update(CurvatureMode=3, AdditionalVolumeMode=2, ConstantsMode=2, UpLiftMode=2, AbortMode=2,
                 MaximumLength=MAX_LENGTH)
    return s


def _planes(field, k):
    p = field.snapshot(k)
    return p, [t.data_ptr() for t in p]


def _engine(c, seed, field, n_snap, **extra):
    precise = c["run"] == "precise"
    e = capi.Engine(capi.settings_from_reference(_reference(c), ring_slots=max(3, n_snap), storage=STORES[c["store"]],
                                                 time_mode=int(precise), compensated=int(precise), **extra))
    for k in range(n_snap):
        keep, ptrs = _planes(field, k)
        torch.cuda.synchronize()
        e.load_windfield_device(k, ptrs, field.shape)
    return e


# ----------------------------------------------------------------- what a program holds before the call

def prepare(c, seed):
    return {"noalloc": _prepare_noalloc, "engine": _prepare_engine, "host": _prepare_host, "batch": _prepare_batch,
            "serve": _prepare_serve}[c["path"]](c, seed)


def _prepare_noalloc(c, seed):
    field = Field(c, seed)
    wind = []
    for k in range(2):
        p = field.snapshot(k)
        zero = [torch.zeros_like(p[0])] if c["dim"] == 3 else []
        wind.append(torch.stack(p + zero, dim=-1).contiguous())
    start = torch.zeros((4, c["n"]), device=DEVICE)
    start[:c["dim"]] = _seeds(c, seed).T
    return dict(c=c, wind=wind, start=start, now=start.clone(),
                settings=capi.settings_from_reference(_reference(c)))


def _prepare_engine(c, seed):
    field, n_snap = Field(c, seed), _snapshots(c)
    e = _engine(c, seed, field, n_snap)
    seeds = _seeds(c, seed)
    e.set_seeds_device(seeds.data_ptr(), c["n"], c["dim"])
    if c["run"] == "plain":
        e.load_volume(0, 0, _temperature(c, seed).cpu().numpy())
        e.compile_expression(0, EXPRESSION, ["T"], [])
    if c["run"] == "general":
        for k in range(n_snap):
            e.load_volume(k, 0, _temperature(c, seed, k).cpu().numpy())
            e.load_constant(k, 0, _constant(c, seed, k).cpu().numpy())
            e.load_uplift(k, _uplift(c, seed, k).cpu().numpy())
        for j, code in enumerate(GENERAL):
            e.compile_expression(j, code, ["T"], ["c"])
    torch.cuda.synchronize()
    return dict(c=c, engine=e, seeds=seeds, n_snap=n_snap)


def _prepare_host(c, seed):
    field, n_snap = Field(c, seed), _snapshots(c)
    page_locked = c["run"] != "gyre"

    def host(t):
        a = pg.pinned_empty(list(t.shape)) if page_locked else np.empty(tuple(t.shape), np.float32)
        a[...] = t.cpu().numpy()
        return a
    wind = [[host(p) for p in field.snapshot(k)] for k in range(n_snap)]
    vols = [{"T": host(_temperature(c, seed))}] if c["run"] == "plain" else []
    values = _reference(c)
    if c["run"] == "plain":
        values["AdditionalCompute"] = [EXPRESSION]
    enums = dict(Space=pg.Space, Integrator=pg.Integrator, WindfieldMode=pg.WindfieldMode, BorderMode=pg.BorderMode,
                 AdditionalVolumeMode=pg.AdditionalVolumeMode, CurvatureMode=pg.CurvatureMode)
    settings = workloads.apply_settings(pg.IntegratorSettings(), values, enums)
    settings.PinnedResults = page_locked
    return dict(c=c, settings=settings, source=workloads.SnapshotSource(wind, volumes=vols),
                seeds=_seeds(c, seed).cpu().numpy())


BATCH_2D = (256, 512)


def _sets(c, seed):
    """Per set: count, lifetime or (start step, steps), and whether it is on the 3D field."""
    rng = np.random.default_rng(1234)        # one mix of sets for every seed
    m = c["sets"]
    counts = np.rint(np.exp(rng.uniform(math.log(max(50, c["n"] // 100)), math.log(c["n"]), m))).astype(int)
    lives = rng.integers(max(2, c["steps"] // 5), c["steps"] + 1, m)
    lives[0] = lives[-1] = c["steps"]        # both fields reach the same last snapshot
    solid = rng.random(m) < 0.7
    solid[0], solid[-1] = True, False
    starts = rng.integers(0, PER_WINDOW * 10, m)
    return counts, lives, solid, starts


def _prepare_batch(c, seed):
    counts, lives, solid, _ = _sets(c, seed)
    n_snap = _snapshots(c)
    groups = []
    for dim, shape in ((3, _shape(c)), (2, BATCH_2D)):
        mine = [j for j in range(c["sets"]) if solid[j] == (dim == 3)]
        d = dict(c, dim=dim, run="positions")
        if dim == 2:
            d.update(nz=1, ny=shape[0], nx=shape[1])
        e = _engine(d, seed + dim, Field(d, seed + dim), n_snap)
        seeds = _seeds(d, seed + dim, n=int(sum(counts[j] for j in mine))).cpu().numpy()
        life = np.concatenate([np.full(counts[j], lives[j], np.int32) for j in mine])
        e.set_seeds(seeds)
        e.set_lifetimes(life)
        groups.append((e, seeds))
    return dict(c=c, groups=groups, batch=capi.Batch([e for e, _ in groups]))


def _serve_snapshots(c):
    return -(-(c["steps"] + PER_WINDOW * 10) // PER_WINDOW) + 1


def _prepare_serve(c, seed):
    counts, lives, _, starts = _sets(c, seed)
    n_snap = _serve_snapshots(c)
    values = dict(_reference(c), MaximumSimulationTime=SPACING * (n_snap - 1))
    server = capi.Server(capi.settings_from_reference(values, storage=STORES[c["store"]]), n_snap, _shape(c),
                         hbm_budget=256 << 20)
    field = Field(c, seed)
    for k in range(n_snap):
        keep, ptrs = _planes(field, k)
        torch.cuda.synchronize()
        server.set_snapshot_device(k, ptrs)
    server.start()
    every = _seeds(c, seed, n=int(counts.sum())).cpu().numpy()
    cut = np.concatenate([[0], np.cumsum(counts)])
    requests = [(every[cut[j]:cut[j + 1]], H * float(starts[j]), int(lives[j])) for j in range(c["sets"])]
    return dict(c=c, server=server, requests=requests)


# ----------------------------------------------------------------- one pass

def run(s):
    c = s["c"]
    if c["path"] == "noalloc":
        now = s["now"]
        now.copy_(s["start"])
        row = [now[k].data_ptr() for k in range(4)]
        done = capi.advance_noalloc(s["settings"], _shape(c), s["wind"][0].data_ptr(), s["wind"][1].data_ptr(), 0.0,
                                    SPACING * max(1, -(-c["steps"] // PER_WINDOW)), 0.0, c["steps"], row[0], row[1],
                                    row[2] if c["dim"] == 3 else None, row[3], c["n"],
                                    torch.cuda.current_stream().cuda_stream)
        return [now[:c["dim"]], now[3].view(torch.int32), done]
    if c["path"] == "engine":
        e = s["engine"]
        e.set_seeds_device(s["seeds"].data_ptr(), c["n"], c["dim"])
        e.run(lambda k: 1 if k < s["n_snap"] else 0)
        if c["save"] == 0:
            return [e.final_positions(), e.status()]
        r = e.results(pinned=True)
        return [r["trajectories"], r["status"], r["lengths"], r["total_curvature"], r["curvatures"],
                r["volume_info"], r["compute_info"]]
    if c["path"] == "host":
        loader = workloads.make_loader(pg.DataLoader, s["source"])
        r = pg.TrajectoryIntegrator(s["settings"], loader, pg.TrajectorySet(s["seeds"])).compute()
        out = [r.trajectories(), r.particleSteps()]
        if c["run"] == "plain":
            out += [r.volumeInfo("T"), r.computeInfo(0)] + ([r.totalCurvatures()] if c["dim"] == 3 else [])
        return out
    if c["path"] == "batch":
        for e, seeds in s["groups"]:
            e.set_seeds(seeds)
        s["batch"].run()
        return [x for e, _ in s["groups"] for x in (e.final_positions(), e.status())]
    server = s["server"]
    ids = [server.submit(*r) for r in s["requests"]]
    out = []
    for rid in ids:
        server.wait(rid)
        p, st, _ = server.result(rid)
        server.release(rid)
        out.append((p, st))
    return [np.concatenate([p for p, _ in out]), np.concatenate([st for _, st in out])]


# ----------------------------------------------------------------- the same in 64 bits

class Sampler:
    """Interpolation in space and time between two snapshots' planes, float64; zero outside the grid in 3D, the
    nearest edge in 2D."""

    def __init__(self, c, scale, off, get):
        self.scale, self.off, self.get, self.dim, self.at, self.tab = scale, off, get, c["dim"], None, None

    def _pad(self, planes):
        x = torch.stack([p.double() for p in planes])
        self.size = list(x.shape[1:])[::-1]
        pad = (1, 2) * self.dim
        if self.dim == 3:
            x = torch.nn.functional.pad(x, pad)
        else:
            x = torch.nn.functional.pad(x[None], pad, mode="replicate")[0]
        return x.reshape(x.shape[0], -1).T

    def window(self, w):
        if w == self.at:
            return
        back = self.front if self.tab is not None and w == self.at + 1 else self._pad(self.get(w))
        self.front = self._pad(self.get(w + 1))
        self.at, self.tab = w, torch.cat([back, self.front], dim=1)

    def __call__(self, p, t):
        lo, frac = [], []
        for d in range(self.dim):
            a = ((p[d] - self.off[d]) / self.scale[d]).clamp(-1.0, float(self.size[d]))
            f = torch.floor(a)
            lo.append(f.long() + 1)
            frac.append((a - f)[:, None])
        row, v = self.size[0] + 3, None
        base = lo[1] * row + lo[0]
        plane = row * (self.size[1] + 3)
        if self.dim == 3:
            base = base + lo[2] * plane

        def along_x(i):
            a = self.tab[i]
            return a + frac[0] * (self.tab[i + 1] - a)

        def along_y(i):
            a = along_x(i)
            return a + frac[1] * (along_x(i + row) - a)
        v = along_y(base)
        if self.dim == 3:
            v = v + frac[2] * (along_y(base + plane) - v)
        m = v.shape[1] // 2
        return [v[:, k] + t * (v[:, m + k] - v[:, k]) for k in range(m)]


def _norm(v):
    return torch.sqrt(sum(x * x for x in v))


def simulate(c, seed, get, seeds, births=None, lives=None, dtd=None, volume=None):
    """The run of `seeds` in float64: records of positions and the other outputs of the engine's results, but for the
    curvatures: they grow as 1 / |v|^2, so a few particles near standstill make the whole of their norm."""
    dim, run_, h = c["dim"], c["run"], _step(c)[0]
    dtd = dtd or _step(c)[1]
    scale, off = _cell(c)
    field = Sampler(c, scale, off, get)
    p = list(seeds.double().T.contiguous())
    n, dev = p[0].numel(), p[0].device
    dom = [_shape(c)[-1 - d] * scale[d] for d in range(dim)]
    zero = torch.zeros(n, dtype=torch.float64, device=dev)
    alive = torch.ones(n, dtype=torch.bool, device=dev)
    length, temp = zero.clone(), zero.clone()
    general, plain = run_ == "general", run_ == "plain"
    vol = Sampler(c, scale, off, volume) if volume else None
    made = [zero.clone() for _ in (GENERAL if general else (EXPRESSION,) if plain else ())]
    records, vols, comps = [torch.stack(p, 1)], [], [[] for _ in made]
    total, per = (c["steps"] if births is None else int((births + lives).max())), dtd / h
    for k in range(total):
        w = int(k // per)
        t = [((k + x) * h - w * dtd) / dtd for x in (0.0, 0.5, 1.0)]
        field.window(w)
        go = alive if births is None else alive & (births <= k) & (k < births + lives)

        def wind(a, tw):
            v = field(a, tw)
            if c["sphere"]:
                v = [v[0] * 180.0 / (_radius(c) * torch.cos(a[1] * (math.pi * 2) / 360.0) * math.pi),
                     v[1] * 180.0 / (math.pi * _radius(c))]
            return v
        v = wind(p, t[0])
        if c["rk4"]:
            k2 = wind([a + 0.5 * h * b for a, b in zip(p, v)], t[1])
            k3 = wind([a + 0.5 * h * b for a, b in zip(p, k2)], t[1])
            k4 = wind([a + h * b for a, b in zip(p, k3)], t[2])
            v = [(a + 2 * b + 2 * d + e) / 6.0 for a, b, d, e in zip(v, k2, k3, k4)]
        step = [x * h for x in v]
        if general:
            b, f = _uplift(c, seed, w).double(), _uplift(c, seed, w + 1).double()
            step = [x + (b[:, d] + t[0] * (f[:, d] - b[:, d])) for d, x in enumerate(step)]
        cut = torch.zeros_like(alive)
        if general:
            size = _norm(step)
            cut = length + size > MAX_LENGTH
            part = torch.where(cut, (MAX_LENGTH - length) / size, torch.ones_like(size))
            step = [x * part for x in step]
            length = torch.where(go, torch.where(cut, torch.full_like(size, MAX_LENGTH), length + size), length)
        new = [a + b for a, b in zip(p, step)]
        still = ~cut & (sum(x * x for x in step) < 1e-9)
        loop = {0: (), 1: (0,), 3: (0, 1)}[c["border"]]
        new = [torch.where(cut | still, x, torch.fmod(x - off[d] + dom[d], dom[d]) + off[d]) if d in loop else x
               for d, x in enumerate(new)]
        out = torch.zeros_like(alive)
        for d in range(dim):
            if d not in loop:
                out = out | (new[d] - off[d] > dom[d]) | (new[d] - off[d] < 0)
        lost = still | (out & ~cut)
        moved = go & ~lost
        p = [torch.where(moved, a, b) for a, b in zip(new, p)]
        if vol is not None:
            vol.window(w if general else 0)
            temp = torch.where(moved, vol(p, t[0] if general else 0.0)[0], temp)
            if general:
                cb, cf = _constant(c, seed, w).double(), _constant(c, seed, w + 1).double()
                values = [torch.sqrt(v[0] ** 2 + v[1] ** 2) * temp + (cb + t[0] * (cf - cb)),
                          temp - 0.5 * v[2] + p[2] * 0.001]
            else:
                values = [torch.sqrt(v[0] ** 2 + v[1] ** 2) * temp]
            made = [torch.where(moved, a, b) for a, b in zip(values, made)]
        alive = alive & ~(go & (lost | cut))
        if c["save"] and k % c["save"] == 0:
            records.append(torch.stack(p, 1))
            if vol is not None:
                vols.append(temp)
                for x, y in zip(comps, made):
                    x.append(y)
    return dict(final=torch.stack(p, 1), records=records, lengths=length, vols=vols, comps=comps)


def exact(c, seed):
    if c["path"] == "batch":
        counts, lives, solid, _ = _sets(c, seed)
        out = []
        for dim, shape in ((3, _shape(c)), (2, BATCH_2D)):
            mine = [j for j in range(c["sets"]) if solid[j] == (dim == 3)]
            d = dict(c, dim=dim, run="positions")
            if dim == 2:
                d.update(nz=1, ny=shape[0], nx=shape[1])
            seeds = _seeds(d, seed + dim, n=int(sum(counts[j] for j in mine)))
            life = torch.as_tensor(np.concatenate([np.full(counts[j], lives[j]) for j in mine]), device=DEVICE)
            r = simulate(d, seed, _stored(d, Field(d, seed + dim)), seeds, torch.zeros_like(life), life)
            out += [r["final"], None]
        return out
    if c["path"] == "serve":
        counts, lives, _, starts = _sets(c, seed)
        births, life = (torch.as_tensor(np.repeat(x, counts), device=DEVICE) for x in (starts, lives))
        r = simulate(c, seed, _stored(c, Field(c, seed)), _seeds(c, seed, n=int(counts.sum())), births, life)
        return [r["final"], None]
    field, seeds = Field(c, seed), _seeds(c, seed)
    if c["path"] == "noalloc":
        r = simulate(c, seed, field.snapshot, seeds, dtd=SPACING * max(1, -(-c["steps"] // PER_WINDOW)))
        return [r["final"].T, None, None]
    volume = None
    if c["run"] == "plain":
        volume = lambda k: [_temperature(c, seed)]  # noqa: E731
    if c["run"] == "general":
        volume = lambda k: [_temperature(c, seed, k)]  # noqa: E731
    r = simulate(c, seed, _stored(c, field), seeds, volume=volume)
    if c["path"] == "host":
        whole = torch.stack(r["records"] + ([r["final"]] if c["save"] == 0 else []), 1)
        out = [whole, None]
        if c["run"] == "plain":
            out += [torch.stack(r["vols"], 1), torch.stack(r["comps"][0], 1)] + [None] * (c["dim"] - 2)
        return out
    if c["save"] == 0:
        return [r["final"], None]
    return [torch.stack(r["records"], 1), None, r["lengths"], None, None,
            [torch.stack(r["vols"], 1)] if r["vols"] else [], [torch.stack(x, 1) for x in r["comps"] if x]]


def _stored(c, field):
    """The snapshots as the storage type of the case rounds them."""
    kind = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[c["store"]]
    return lambda k: [p.to(kind).float() for p in field.snapshot(k)]


# ----------------------------------------------------------------- what a pass cannot do without

def work(c):
    """Each snapshot read once (no more of it than the particles sample), seeds read, results written; the
    interpolations of every step: 7 (3) lerps a component and snapshot, one in time, 3 operations each."""
    dim = c["dim"]
    nodes = c["nz"] * c["ny"] * c["nx"]
    per_node = dim * (4 if c["store"] == "f32" or c["path"] in ("noalloc", "host") else 2)
    stages, lerps = 4 if c["rk4"] else 1, 7 if dim == 3 else 3
    n, steps = c["n"], c["steps"]
    snaps = 2 if c["path"] == "noalloc" else _snapshots(c)
    if c["path"] in ("batch", "serve"):
        counts, lives, _, _ = _sets(c, 0)
        n, steps = int(counts.sum()), float((counts * lives).sum()) / float(counts.sum())
        snaps = _serve_snapshots(c) if c["path"] == "serve" else snaps
    flops = n * steps * (stages * dim * (2 * lerps + 1) * 3 + 20 * dim)
    touched = min(nodes, n * 2 ** dim * (1 + min(PER_WINDOW, steps)))
    saves = 1 + -(-c["steps"] // c["save"]) if c["save"] else 1
    extra = {"plain": 2, "general": 4}.get(c["run"], 0)
    wrote = n * 4 * (saves * dim + (saves - 1) * extra + 1)
    read = snaps * touched * per_node + n * 4 * dim
    if c["run"] == "general":
        read += snaps * (nodes * 4 + n * 16)
    elif extra:
        read += nodes * 4
    return {"bytes": float(read + wrote), "flops": float(flops)}
