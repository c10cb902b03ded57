"""The solver's performance cases: what programs on this framework have it do.

A case is a dict of plain values with a ``kind``:

* ``sort``   the stable neighbour-grid counting sort (pf_sort) on device buffers
* ``dam``    one fluid scene (dam break in an open tank), a frame and its readback
* ``surface`` one fluid scene with the facade's default surface effects
* ``mixed``  fluid, soft bodies and a moving sphere in one scene
* ``pile``   soft bodies falling on each other, particle contacts on
* ``cloth``  one hanging sheet: stretch, bending, tethers, wind, smoothing
* ``batch``  uneven scenes packed into one world (pf_batch), positions read every frame
* ``bake``   a triangle mesh baked into a signed-distance grid

One pass of a scene is one frame (1/60 s) of a running simulation and the read
of its state, so a state moves on from pass to pass.
"""

from __future__ import annotations

import ctypes as C
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "threejs-particle-fluids_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from pfsim import _native as N  # noqa: E402
from pfsim import api  # noqa: E402
from pfsim import hashgrid as H  # noqa: E402
from pfsim import mesh as M  # noqa: E402
from pfsim import recipe as R  # noqa: E402
from pfsim import workloads as W  # noqa: E402

DT = 1.0 / 60.0
TANK = ((-0.5, 0.0, -0.3), (0.5, 0.8, 0.3))
BLOCK = ((-0.5, 0.0, -0.3), (-0.1, 0.5, 0.3))


# ------------------------------------------------------------------ cases ----
def listed() -> list[dict]:
    return [
        # the neighbour search of one interactive scene, in the reference's
        # Morton buckets: the smallest call, where launches count
        {"name": "sort_morton_20k", "kind": "sort", "n": 20_011, "keys": "morton", "dist": "uniform"},
        # a large scene's particles, clustered as a fluid's are, an odd count
        {"name": "sort_blobs_1m", "kind": "sort", "n": 1_000_003, "keys": "linear", "dist": "blobs"},
        # the largest sort: 16M particles on a 128^3 grid
        {"name": "sort_uniform_16m", "kind": "sort", "n": 16_000_000, "keys": "linear", "dist": "uniform"},
        # the default interactive scene: 5,000 fluid particles, stepped alone
        {"name": "dam_5k", "kind": "dam", "n": 5_000},
        # a fluid scene at the top of the batch's size range, stepped alone
        {"name": "dam_200k", "kind": "dam", "n": 200_000},
        # the facade's fluid: XSPH, vorticity confinement, surface tension,
        # adhesion, the substeps the facade gives that particle size
        {"name": "surface_30k", "kind": "surface", "n": 30_000},
        # fluid coupled with 20 soft bodies and a swept sphere
        {"name": "mixed_50k", "kind": "mixed", "n": 50_000},
        # 100 soft bodies piling up with particle contacts
        {"name": "pile_50k", "kind": "pile", "n": 50_000},
        # a full cloth: every cloth term the library has
        {"name": "cloth_256", "kind": "cloth", "side": 256},
        # offline batching: many uneven fluid and cloth scenes in one world
        {"name": "batch_96", "kind": "batch", "scenes": 96, "lo": 5_000, "hi": 200_000, "fluid": 0.7, "soft": 0.0,
         "stream": 0},
        # what a serving tick steps: fluid, soft bodies and cloth together
        {"name": "cohort_24", "kind": "batch", "scenes": 24, "lo": 5_000, "hi": 200_000, "fluid": 0.6, "soft": 0.2,
         "stream": 7},
        # scene set-up: a mesh of about 4,000 triangles into a 128^3 field
        {"name": "bake_128", "kind": "bake", "res": 128, "segments": 64},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["sort", "sort", "dam", "dam", "surface", "mixed", "pile", "cloth", "batch", "batch", "bake"])
    if kind == "sort":
        return {"kind": kind, "n": int(_log(rng, 4_000, 16_000_000)), "keys": rng.choice(["linear", "morton"]),
                "dist": rng.choice(["uniform", "blobs"])}
    if kind == "dam":
        return {"kind": kind, "n": int(_log(rng, 5_000, 200_000))}
    if kind == "surface":
        return {"kind": kind, "n": int(_log(rng, 5_000, 60_000))}
    if kind == "mixed":
        return {"kind": kind, "n": int(_log(rng, 10_000, 50_000))}
    if kind == "pile":
        return {"kind": kind, "n": int(_log(rng, 10_000, 50_000))}
    if kind == "cloth":
        return {"kind": kind, "side": rng.randint(64, 256)}
    if kind == "batch":
        soft = rng.choice([0.0, 0.2])
        return {"kind": kind, "scenes": int(_log(rng, 4, 48 if soft == 0.0 else 24)), "lo": 5_000, "hi": 200_000,
                "fluid": 0.7 if soft == 0.0 else 0.6, "soft": soft, "stream": rng.randrange(1 << 20)}
    return {"kind": kind, "res": rng.randint(32, 128), "segments": rng.randint(16, 64)}


# ----------------------------------------------------------------- inputs ----
def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _sort_positions(case: dict, seed: int) -> torch.Tensor:
    g, n = _generator(seed), case["n"]
    pos = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    if case["dist"] == "uniform":
        pos[:, :3] = torch.rand((n, 3), generator=g, device="cuda")
    else:  # 64 Gaussian blobs (sigma 0.02), clamped into the unit cube
        centres = torch.rand((64, 3), generator=g, device="cuda")
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        pts = centres[which] + 0.02 * torch.randn((n, 3), generator=g, device="cuda")
        pos[:, :3] = pts.clamp_(0.0, 1.0 - 2.0**-24)
    return pos


def _sort_grid(case: dict) -> H.GridOptions:
    if case["keys"] == "linear":
        return H.GridOptions(cell_size=W.SORT_CELL, kind="linear", dims=W.SORT_GRID_DIMS)
    # about eight particles a cell, as a fluid's smoothing radius gives
    return H.GridOptions(cell_size=2.0 * case["n"] ** (-1.0 / 3.0), kind="morton")


def _with_velocities(rec: R.Recipe, seed: int) -> R.Recipe:
    """The recipe's uploads with seeded velocities (normal, 0.1 m/s)."""
    g = np.random.default_rng(seed)
    for u in rec.uploads:
        u.vel = g.normal(0.0, 0.1, (len(u.pos), 3)).astype(np.float32)
    return rec


def _surface_recipe(case: dict, seed: int) -> R.Recipe:
    lo, hi = np.array(BLOCK[0]), np.array(BLOCK[1])
    s = float(np.prod(hi - lo) / case["n"]) ** (1.0 / 3.0)
    h, mass = 2.0 * s, 1000.0 * s**3
    pts = W.fill_box(lo, hi, s)
    pts = pts + np.random.default_rng(seed).uniform(-0.05 * s, 0.05 * s, pts.shape)
    rho0 = W.lattice_rest_density(s, h, mass)
    fluid = R.FluidOpts(range=(0, len(pts)), rest_density=rho0, particle_spacing=(mass / rho0) ** (1.0 / 3.0),
                        smoothing_radius=h, compliance=1e-4, viscosity=0.01, vorticity=0.02, surface_tension=0.1,
                        adhesion=0.1)
    tlo, thi = np.array(TANK[0]), np.array(TANK[1])
    loop = R.LoopOpts(substeps=min(24, math.ceil(4 * max(1.0, 0.018 / (0.5 * s)))), iterations=2,
                      grid_min=tuple(tlo - 2 * h), grid_max=tuple(thi + np.array([2 * h, 0.8, 2 * h])))
    return R.Recipe(capacity=len(pts), radius=0.5 * s, uploads=[R.Upload(0, pts.astype(np.float32))],
                    materials=[("fluid", fluid)], prims=R.container_walls(*TANK), loop=loop)


def _recipe(case: dict, seed: int) -> R.Recipe:
    kind = case["kind"]
    if kind == "dam":
        return W.dam_break(case["n"], seed=seed)
    if kind == "surface":
        return _surface_recipe(case, seed)
    if kind == "mixed":
        return _with_velocities(W.mixed_scene(case["n"], n_fluid=3 * case["n"] // 5), seed)
    if kind == "pile":
        rec = _with_velocities(W.softbody_pile(case["n"], per_body=500), seed)
        rec.loop.contact = True
        return rec
    return W.cloth_sheet(case["side"], seed=seed, bend_compliance=1e-5, tethers=True, stretch_tolerance=0.06,
                         wind=(0.8, 0.0, 1.5), drag=0.18, lift=0.02, damping=0.1)


def _stream(case: dict) -> list[tuple[str, int, float]]:
    """(material, particles, container scale) of each scene of a batch."""
    r = random.Random(case["stream"])
    out = []
    for _ in range(case["scenes"]):
        n, u, scale = int(_log(r, case["lo"], case["hi"])), r.random(), r.uniform(0.5, 2.0)
        out.append(("fluid" if u < case["fluid"] else "soft" if u < case["fluid"] + case["soft"] else "cloth", n, scale))
    return out


def _batch_recipes(case: dict, seed: int) -> list[R.Recipe]:
    out = []
    for i, (what, n, scale) in enumerate(_stream(case)):
        s = 1009 * seed + i
        if what == "fluid":
            out.append(W.dam_break(n, seed=s, scale=scale))
        elif what == "soft":
            out.append(_with_velocities(W.softbody_pile(n, seed=i, scale=scale, substeps=2), s))
        else:
            out.append(W.cloth_sheet(min(256, max(64, round(math.sqrt(n)))), seed=s, scale=scale))
    return out


def _mesh(case: dict, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """A bumpy closed surface, turned and dented by the seed."""
    v, idx = M.uv_sphere(0.5, case["segments"], case["segments"])
    r = np.random.default_rng(seed)
    q, _ = np.linalg.qr(r.normal(size=(3, 3)))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    waves, phase = r.normal(0.0, 4.0, (3, 3)), r.uniform(0.0, 6.28, 3)
    bump = 1.0 + 0.08 * np.sin(v.astype(np.float64) @ waves.T + phase).sum(1)
    return ((v * bump[:, None]) @ q.T).astype(np.float32), idx


# ------------------------------------------------------------ entry points ----
class _Scene:
    """A scene handle and the frame it is at."""

    def __init__(self, rec: R.Recipe):
        self.scene = R.NativeBackend().build(rec)

    def run(self):
        self.scene.step(DT)
        return {"positions": self.scene.readback(N.PF_FIELD_POSITIONS),
                "velocities": self.scene.readback(N.PF_FIELD_VELOCITIES)}


class _Batch:
    """A batch and two pinned host buffers its positions go to in turn."""

    def __init__(self, recs: list[R.Recipe]):
        scenes = [R.NativeBackend().build(r) for r in recs]
        self.batch = R.Batch(scenes)
        for s in scenes:
            s.close()
        total = sum(r.capacity for r in recs)
        self.host = [torch.empty((total, 4), dtype=torch.float32, pin_memory=True) for _ in range(2)]
        self.turn = 0

    def run(self):
        out = self.host[self.turn]
        self.turn ^= 1
        self.batch.step(DT)
        N.check(N.lib().pf_batch_read_positions_async(self.batch.h, C.cast(out.data_ptr(), C.POINTER(C.c_float)),
                                                      out.numel() * 4))
        return out


class _Sort:
    """Positions, the grid and the buffers a frame loop sorts into."""

    def __init__(self, case: dict, seed: int):
        self.n = case["n"]
        self.pos = _sort_positions(case, seed)
        self.desc = _sort_grid(case).desc(self.n)
        cells = int(N.lib().pf_grid_cells(C.byref(self.desc)))
        new = lambda k: torch.empty(k, dtype=torch.int32, device="cuda")  # noqa: E731
        self.out = {"perm": new(self.n), "start": new(cells), "count": new(cells), "keys": new(self.n),
                    "overflow": new(1)}

    def run(self):
        p = {k: C.c_void_p(t.data_ptr()) for k, t in self.out.items()}
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        N.check(N.lib().pf_sort(C.c_void_p(self.pos.data_ptr()), self.n, C.byref(self.desc), p["perm"], p["start"],
                                p["count"], p["keys"], p["overflow"], stream))
        return self.out


class _Bake:
    def __init__(self, case: dict, seed: int):
        self.mesh, self.res = _mesh(case, seed), case["res"]

    def run(self):
        data, origin, voxel, split = M.bake_sdf(*self.mesh, self.res)
        return {"data": data, "origin": origin, "voxel": float(voxel), "split": int(split)}


def prepare(case: dict, seed: int):
    if case["kind"] == "sort":
        return _Sort(case, seed)
    if case["kind"] == "bake":
        return _Bake(case, seed)
    if case["kind"] == "batch":
        return _Batch(_batch_recipes(case, seed))
    return _Scene(_recipe(case, seed))


def run(state):
    return state.run()


# ------------------------------------------------------------------- work ----
def _fluid_work(n: int, substeps: int, iterations: int) -> tuple[float, float]:
    # position and velocity in and out once a frame; about 33 neighbours, 15
    # operations each, in the density and position sums and XSPH
    return 64.0 * n, float(substeps) * n * 33 * 15 * (2 * iterations + 1)


def _soft_work(n: int, substeps: int, iterations: int) -> tuple[float, float]:
    # with the orientation; about 20 members a cluster, 60 operations each
    return 128.0 * n, float(substeps) * iterations * n * (20 * 60 + 600)


def _cloth_work(n: int, substeps: int, iterations: int, full: bool) -> tuple[float, float]:
    # 3 edges a particle, with bending 3 hinges, a tether and 6 triangles
    return 64.0 * n, float(substeps) * n * (iterations * (3 * 25 + (3 * 200 + 25 if full else 0)) + (600 if full else 0))


def work(case: dict) -> dict:
    kind, n = case["kind"], case.get("n", 0)
    if kind == "sort":
        cells = 128**3 if case["keys"] == "linear" else 1 << (2 * n - 1).bit_length()
        b, f = 24.0 * n + 8.0 * cells, 0.0
    elif kind == "dam":
        b, f = _fluid_work(n, 2, 4)
    elif kind == "surface":
        s = (0.12 / n) ** (1.0 / 3.0)
        sub = min(24, math.ceil(4 * max(1.0, 0.036 / s)))
        b, f = _fluid_work(n, sub, 2)
        f += sub * n * 33 * 60.0
    elif kind == "mixed":
        b0, f0 = _fluid_work(3 * n // 5, 3, 4)
        b1, f1 = _soft_work(n - 3 * n // 5, 3, 4)
        b, f = b0 + b1, f0 + f1
    elif kind == "pile":
        b, f = _soft_work(n, 3, 4)
        f += 3.0 * n * (27 * 10 + 4 * 4 * 60)
    elif kind == "cloth":
        b, f = _cloth_work(case["side"] ** 2, 2, 4, True)
    elif kind == "batch":
        b = f = 0.0
        for what, m, _ in _stream(case):
            side = min(256, max(64, round(math.sqrt(m))))
            x = (_fluid_work(m, 2, 4) if what == "fluid" else _soft_work(m, 2, 4) if what == "soft"
                 else _cloth_work(side * side, 2, 4, False))
            b, f = b + x[0], f + x[1]
    else:
        # per voxel the closest triangle of a few, three ray parities
        b, f = 4.0 * case["res"] ** 3 + 72.0 * case["segments"] ** 2, 300.0 * case["res"] ** 3
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- 64-bit restatement ----
def _f64(a, device) -> torch.Tensor:
    return torch.as_tensor(np.asarray(a, np.float64), device=device)


class _Walls:
    """Static planes with friction against particles of one radius: the
    contact of each substep's iterations, then its kinetic friction."""

    def __init__(self, rec: R.Recipe, n: int, device):
        self.radius = rec.radius
        self.planes = [(_f64(p.data0[:3], device), _f64(p.data1[:3], device), p.data1[3], p.velocity[3])
                       for p in rec.prims]
        self.ln = torch.zeros((len(self.planes), n), dtype=torch.float64, device=device)
        self.lt = torch.zeros_like(self.ln)

    def reset(self):
        self.ln.zero_()
        self.lt.zero_()

    def solve(self, xs, x, w):
        move = torch.zeros_like(xs)
        for k, (nrm, at, mu_s, _) in enumerate(self.planes):
            phi = (xs - at) @ nrm
            hit = (phi < self.radius) & (w > 0)
            depth = torch.where(hit, self.radius - phi, torch.zeros_like(phi))
            safe_w = torch.where(w > 0, w, torch.ones_like(w))
            ln = self.ln[k] + depth / safe_w
            slip = xs - x
            tang = slip - nrm * (slip @ nrm)[:, None]
            tl = tang.norm(dim=1)
            stick = hit & (tl > 1e-10) & (tl / safe_w <= mu_s * ln - self.lt[k])
            move += depth[:, None] * nrm - torch.where(stick[:, None], tang, torch.zeros_like(tang))
            self.ln[k] = ln
            self.lt[k] += torch.where(stick, tl / safe_w, torch.zeros_like(tl))
        return xs + move

    def friction(self, v, w, dt):
        out = v.clone()
        for k, (nrm, _, _, mu_k) in enumerate(self.planes):
            vt = v - nrm * (v @ nrm)[:, None]
            vl = vt.norm(dim=1)
            change = torch.minimum(mu_k * self.ln[k] * w / dt, vl)
            go = (self.ln[k] > 0) & (vl > 1e-6)
            out -= torch.where(go[:, None], vt / vl.clamp_min(1e-30)[:, None] * change[:, None], torch.zeros_like(vt))
        return out


def _pairs(x: torch.Tensor, h: float) -> tuple[torch.Tensor, torch.Tensor]:
    """Every ordered pair (i, j), i itself among them, within h."""
    cell = torch.floor(x / h).long()
    cell -= cell.amin(0) - 1
    dims = cell.amax(0) + 2
    flat = lambda c: (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]  # noqa: E731
    key, order = torch.sort(flat(cell))
    ii, jj = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                want = flat(cell + torch.tensor([dx, dy, dz], device=x.device))
                lo, hi = torch.searchsorted(key, want), torch.searchsorted(key, want, right=True)
                cnt = hi - lo
                i = torch.repeat_interleave(torch.arange(len(x), device=x.device), cnt)
                off = torch.arange(len(i), device=x.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
                j = order[lo[i] + off]
                near = ((x[i] - x[j]) ** 2).sum(1) < h * h
                ii.append(i[near])
                jj.append(j[near])
    return torch.cat(ii), torch.cat(jj)


def _exact_dam(rec: R.Recipe, device) -> dict:
    f = rec.materials[0][1]
    n, h, rho0 = rec.capacity, f.smoothing_radius, f.rest_density
    m = rho0 * f.particle_spacing**3
    w = torch.full((n,), 1.0 / m, dtype=torch.float64, device=device)
    x = _f64(rec.uploads[0].pos, device)
    v = torch.zeros_like(x)
    g = _f64(rec.loop.gravity, device)
    dt = DT / rec.loop.substeps
    walls = _Walls(rec, n, device)
    poly6 = lambda r2: 315.0 / (64.0 * math.pi * h**9) * (h * h - r2).clamp_min(0.0) ** 3  # noqa: E731
    add = lambda i, t: torch.zeros((n, *t.shape[1:]), dtype=t.dtype, device=device).index_add_(0, i, t)  # noqa: E731

    def gradient(d):
        r = d.norm(dim=1)
        return d * (-45.0 / (math.pi * h**6) * (h - r).clamp_min(0.0) ** 2 / r.clamp_min(1e-20))[:, None]

    for _ in range(rec.loop.substeps):
        v = v + g * dt
        xs = x + v * dt
        walls.reset()
        i, j = _pairs(xs, h)
        for _ in range(rec.loop.iterations):
            d = xs[i] - xs[j]
            grad = gradient(d)
            rho = add(i, m * poly6((d * d).sum(1)))
            gs = add(i, m * grad)
            gss = add(i, (m * m) * (grad * grad).sum(1) * w[j])
            c = rho / rho0 - 1.0
            den = ((gs * gs).sum(1) * w + gss) / rho0**2 + f.compliance / dt**2
            lam = torch.where(c > 0, -c / den, torch.zeros_like(c))
            xs = xs + add(i, grad * ((lam[i] + lam[j]) * m)[:, None]) / rho0 * w[:, None]
            xs = walls.solve(xs, x, w)
        v, x = (xs - x) / dt, xs
        d = x[i] - x[j]
        v = v + f.viscosity * add(i, (v[j] - v[i]) * (poly6((d * d).sum(1)) * f.particle_spacing**3)[:, None])
        v = walls.friction(v, w, dt)
    return _rows(x, v)


def _rows(x, v) -> dict:
    pad = lambda t: torch.cat([t, torch.zeros_like(t[:, :1])], 1)  # noqa: E731
    return {"positions": pad(x), "velocities": pad(v)}


def _colours(parts: np.ndarray) -> list[np.ndarray]:
    """Constraints grouped so that no two of a group share a particle: each
    takes the lowest group its particles are not in yet, in order."""
    used = [0] * (int(parts.max()) + 1)
    group = np.empty(len(parts), np.int64)
    for c, row in enumerate(parts.tolist()):
        mask = 0
        for p in row:
            mask |= used[p]
        bit = ~mask & (mask + 1)
        for p in row:
            used[p] |= bit
        group[c] = bit.bit_length() - 1
    return [np.flatnonzero(group == k) for k in range(group.max() + 1)]


def _exact_cloth(rec: R.Recipe, device) -> dict:
    o = rec.materials[0][1]
    x, w = _f64(o.positions, device), _f64(o.inv_mass, device)
    n, v = len(x), torch.zeros_like(x)
    idx = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=device)  # noqa: E731
    pairs, bends, tris = idx(o.pairs), idx(o.bending), idx(o.triangles)
    tie = torch.stack([idx(o.tether_particle), idx(o.tether_anchor)], 1)
    rest, angle, reach = _f64(o.rest_lengths, device), _f64(o.bending_rest, device), _f64(o.tether_rest, device)
    pair_groups = [idx(c) for c in _colours(np.asarray(o.pairs))]
    bend_groups = [idx(c) for c in _colours(np.asarray(o.bending))]
    tie_groups = [idx(c) for c in _colours(np.asarray(o.tether_particle)[:, None])]
    dt = DT / rec.loop.substeps
    g, wind = _f64(rec.loop.gravity, device), _f64(o.wind, device)
    free = (w > 0)[:, None]
    walls = _Walls(rec, n, device)
    add = lambda i, t: torch.zeros((n, *t.shape[1:]), dtype=t.dtype, device=device).index_add_(0, i, t)  # noqa: E731
    dot = lambda a, b: (a * b).sum(1)  # noqa: E731
    cross = lambda a, b: torch.linalg.cross(a, b)  # noqa: E731
    degree = add(pairs.reshape(-1), torch.ones(2 * len(pairs), dtype=torch.float64, device=device)).clamp_min(1.0)

    def stretch(xs, lam, c):
        i, j = pairs[c, 0], pairs[c, 1]
        d = xs[i] - xs[j]
        l, ws, at = d.norm(dim=1), w[i] + w[j], o.stretch_compliance / dt**2
        dl = torch.where((ws > 0) & (l >= 1e-12), (-(l - rest[c]) - at * lam[c]) / (ws + at), torch.zeros_like(l))
        lam[c] += dl
        nrm = d / l.clamp_min(1e-12)[:, None]
        xs[i] += nrm * (w[i] * dl)[:, None]
        xs[j] -= nrm * (w[j] * dl)[:, None]

    def bend(xs, lam, c):
        p = bends[c]
        x1, x2, x3, x4 = (xs[p[:, k]] for k in range(4))
        e = x2 - x1
        el = e.norm(dim=1)
        n1, n2 = cross(x3 - x1, x3 - x2), cross(x4 - x2, x4 - x1)
        s1, s2 = dot(n1, n1), dot(n2, n2)
        ok = (el * el >= 1e-24) & (s1 >= 1e-24) & (s2 >= 1e-24)
        a, b, el = n1 / s1.clamp_min(1e-24)[:, None], n2 / s2.clamp_min(1e-24)[:, None], el.clamp_min(1e-12)
        err = torch.atan2(dot(cross(n1, n2), e), dot(n1, n2) * el) - angle[c]
        part = lambda u, t: u * (dot(t, e) / el)[:, None]  # noqa: E731
        grads = [-(part(a, x3 - x2) + part(b, x4 - x2)), part(a, x3 - x1) + part(b, x4 - x1),
                 -a * el[:, None], -b * el[:, None]]
        sg = sum(dot(q, q) * w[p[:, k]] for k, q in enumerate(grads))
        at = o.bend_compliance / dt**2
        dl = torch.where(ok & (sg > 1e-30), (-err - at * lam[c]) / (sg + at), torch.zeros_like(sg))
        lam[c] += dl
        for k, q in enumerate(grads):
            xs[p[:, k]] += q * (w[p[:, k]] * dl)[:, None]

    def tether(xs, lam, c):
        i = tie[c, 0]
        d = xs[i] - xs[tie[c, 1]]
        l, at = d.norm(dim=1), o.tether_compliance / dt**2
        on = (l > reach[c]) & (w[i] > 0)
        dl = torch.where(on, (-(l - reach[c]) - at * lam[c]) / (w[i] + at).clamp_min(1e-30), torch.zeros_like(l))
        lam[c] = torch.where(on, lam[c] + dl, torch.zeros_like(l))
        xs[i] += d / l.clamp_min(1e-12)[:, None] * (w[i] * dl)[:, None]

    for _ in range(rec.loop.substeps):
        v = torch.where(free, v + g * dt, v)
        xs = torch.where(free, x + v * dt, x)
        walls.reset()
        t1, t2, t3 = tris.T
        vrel = (v[t1] + v[t2] + v[t3]) / 3.0 - wind
        raw = cross(x[t2] - x[t1], x[t3] - x[t1])
        speed, area2 = vrel.norm(dim=1), raw.norm(dim=1)
        go = (speed * speed > 1e-12) & (area2 * area2 > 1e-12)
        nu, vh = raw / area2.clamp_min(1e-30)[:, None], vrel / speed.clamp_min(1e-30)[:, None]
        nb = nu * torch.where(dot(nu, vrel) < 0, -1.0, 1.0)[:, None]
        push = (speed * speed * area2 * 0.5)[:, None]
        force = -vh * (o.drag * dot(nb, vh))[:, None] * push + cross(cross(nb, vh), vh) * o.lift * push
        force = torch.where(go[:, None], force / 3.0, torch.zeros_like(force))
        xs = xs + sum(add(t, force) for t in (t1, t2, t3)) * (dt * dt * w)[:, None]
        lam = [torch.zeros(len(t), dtype=torch.float64, device=device) for t in (pairs, bends, tie)]
        for _ in range(rec.loop.iterations):
            for groups, solve, l in ((pair_groups, stretch, lam[0]), (bend_groups, bend, lam[1]),
                                     (tie_groups, tether, lam[2])):
                for c in groups:
                    solve(xs, l, c)
            xs = walls.solve(xs, x, w)
        v, x = torch.where(free, (xs - x) / dt, v), torch.where(free, xs, x)
        mean = (add(pairs[:, 0], v[pairs[:, 1]]) + add(pairs[:, 1], v[pairs[:, 0]])) / degree[:, None]
        v = torch.where(free, v * (1.0 - o.damping) + mean * o.damping, v)
        v = walls.friction(v, w, dt)
    return _rows(x, v)


def _point_triangle(p: torch.Tensor, a, b, c) -> torch.Tensor:
    """Squared distances of points (n, 1, 3) to triangles (1, t, 3): the best
    of the three edges and, above the face, the plane."""
    dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
    best = None
    for s, e in ((a, b), (b, c), (c, a)):
        d = e - s
        q = p - s
        t = (dot(q, d) / dot(d, d).clamp_min(1e-300)).clamp(0.0, 1.0)
        q = q - t[..., None] * d
        best = dot(q, q) if best is None else torch.minimum(best, dot(q, q))
    nrm = torch.linalg.cross(b - a, c - a, dim=-1)
    over = torch.ones_like(best, dtype=torch.bool)
    for s, e in ((a, b), (b, c), (c, a)):
        over &= (p * (side := torch.linalg.cross(nrm, e - s, dim=-1))).sum(-1) >= dot(s, side)
    high = dot(p - a, nrm)
    return torch.where(over, high * high / dot(nrm, nrm).clamp_min(1e-300), best)


def _exact_bake(case: dict, seed: int, device):
    v, idx = _mesh(case, seed)
    res = case["res"]
    tri = _f64(v, device)[torch.as_tensor(idx.astype(np.int64), device=device)].reshape(-1, 3, 3)
    lo, hi = tri.amin((0, 1)), tri.amax((0, 1))
    k = 2 if res >= 8 else 1
    pad = k * (hi - lo).max() / (res - 2 * k)
    side = (hi - lo).max() + 2 * pad
    voxel, origin = side / res, 0.5 * (lo + hi) - 0.5 * side
    axis = (torch.arange(res, dtype=torch.float64, device=device) + 0.5) * voxel
    a, b, c = (tri[None, :, q] for q in range(3))
    out = torch.empty((res, res, res), dtype=torch.float64, device=device)
    # the winding number of a closed surface is 1 inside and 0 outside
    rows = max(1, 30_000_000 // (res * len(tri)))
    flat = out.view(res * res, res)
    for r0 in range(0, res * res, rows):
        r = torch.arange(r0, min(r0 + rows, res * res), device=device)
        pts = torch.stack([axis.expand(len(r), res), axis[r % res][:, None].expand(-1, res),
                           axis[r // res][:, None].expand(-1, res)], -1) + origin
        p = pts.reshape(-1, 1, 3)
        dist = _point_triangle(p, a, b, c).amin(1).sqrt()
        u, q, s = a - p, b - p, c - p
        lu, lq, ls = u.norm(dim=-1), q.norm(dim=-1), s.norm(dim=-1)
        det = (u * torch.linalg.cross(q, s, dim=-1)).sum(-1)
        den = lu * lq * ls + (u * q).sum(-1) * ls + (q * s).sum(-1) * lu + (s * u).sum(-1) * lq
        wind = torch.atan2(det, den).sum(1) / (2.0 * math.pi)
        flat[r0:r0 + len(r)] = torch.where(wind.abs() > 0.5, -dist, dist).view(len(r), res)
    return {"data": out, "origin": origin.cpu().numpy(), "voxel": float(voxel), "split": None}


def exact(case: dict, seed: int):
    """One frame (or field) in 64 bits. None for the sorts, whose outputs are
    whole numbers, and for scenes with surface effects, soft bodies or many
    scenes, whose thousands of coupled small solves take minutes here."""
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["kind"] == "bake":
        return _exact_bake(case, seed, device)
    if case["kind"] == "dam":
        return _exact_dam(_recipe(case, seed), device)
    if case["kind"] == "cloth":
        return _exact_cloth(_recipe(case, seed), device)
    return None
