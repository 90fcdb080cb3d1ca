"""The work a user of this library has it do, as cases that can be timed and compared.

A pass of every fluid case is a rollout: the caller's state is written to the handle, one or
more ticks are stepped with the reactions read after each, and the resulting state is read
back into the caller's (pinned) buffers. Starting each pass from the caller's state keeps a
pass the same work however often it runs; the constants of the large scenes are acoustically
stiff (see _stiff), and a scene left running would spread over a grid no dam break occupies.

prepare() builds the scene and its handle (the device pool, the uploaded particles), run() is
one rollout, exact() the same rollout in 64-bit torch without the library.
"""
from __future__ import annotations

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
for _p in (ROOT, ROOT / "rust-wl_b200"):
    if str(_p) not in sys.path:
        sys.path.insert(0, str(_p))

import vxl_sph  # noqa: E402
from vxl_sph import scenes  # noqa: E402

F32 = np.float32
DT = float(F32(1.0) / F32(60.0))  # 60 Hz ticks
GRAVITY = (0.0, -9.81, 0.0)


def listed():
    return [
        # the smallest scene a frame loop steps: 512 particles in an Akinci tank, one tick; launches and host calls
        dict(name="tiny_tick", kind="tick", nx=8, ny=8, nz=8, s=0.05, tx=0.6, ty=0.5, tz=0.5, sub=4, ticks=1,
             disorder=0.01, u0=0.0, boxes=0),
        # dam0, the 16k dam break: the usual interactive size
        dict(name="dam0_tick", kind="tick", nx=16, ny=32, nz=32, s=0.02, tx=1.0, ty=0.64, tz=0.64, sub=10, ticks=1,
             disorder=0.01, u0=0.0, boxes=0),
        # the reference's stepper loop: the caller moves its bodies and re-uploads the boundary segment every tick
        dict(name="stepper_moving", kind="stepper", nx=31, ny=37, nz=29, s=0.02, tx=0.9, ty=1.0, tz=0.6, sub=20, ticks=3,
             disorder=0.1, u0=0.4, boxes=3),
        # the reference's grid probe: a free 50^3 lattice with the default configuration, no walls
        dict(name="probe_block", kind="block", nx=50, ny=50, nz=50, s=0.05, sub=4, ticks=2, disorder=0.01, u0=0.0),
        # provider walls (five tank faces and a convex obstacle) instead of boundary particles
        dict(name="provider_tank", kind="walls", nx=41, ny=37, nz=43, s=0.02, tx=1.6, ty=1.2, tz=0.86, sub=10, ticks=1,
             disorder=0.1, u0=0.5),
        # floating boxes integrated on the device between ticks
        dict(name="coupled_boxes", kind="coupled", nx=47, ny=43, nz=39, s=0.02, tx=1.2, ty=1.2, tz=0.8, sub=20, ticks=2,
             disorder=0.05, u0=0.3, boxes=6),
        # dam1, the 1M dam break, from its initial lattice
        dict(name="dam1_tick", kind="tick", nx=100, ny=100, nz=100, s=0.01, tx=2.0, ty=2.0, tz=1.0, sub=10, ticks=1,
             disorder=0.01, u0=0.0, boxes=0),
        # a flowing, odd-sized pool in a wide tank: the cell budget doubles the bins to 2h
        dict(name="wide_pool", kind="tick", nx=173, ny=53, nz=149, s=0.005, tx=2.5, ty=1.2, tz=1.2, sub=10, ticks=1,
             disorder=0.1, u0=0.5, boxes=0),
        # dam10m, the headline scene: 9.94M fluid particles, walls and 64 boxes
        dict(name="dam10m_tick", kind="tick", nx=215, ny=215, nz=215, s=0.005, tx=2.5, ty=1.2, tz=1.2, sub=10, ticks=1,
             disorder=0.01, u0=0.0, boxes=64),
        # uneven tanks (4k to 262k) stepped together in one handle
        dict(name="batch_tanks", kind="batch", scenes=32, lo=4096, hi=262144, mix=7, sub=10, ticks=2),
        # requests served with continuous batching: submitted together, stepped until all are done, read
        dict(name="serve_requests", kind="serve", scenes=12, lo=8192, hi=131072, mix=11, sub=10, ticks=2),
        # the neighbour table alone, built into the caller's device buffers
        dict(name="grid_table", kind="grid", nx=83, ny=71, nz=73, s=0.01, bins=524288, disorder=0.1),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def dims(n):
        a, b = log(0.4, 2.5), log(0.5, 2.0)
        nx = max(3, round((n * a * a / b) ** (1 / 3)))
        ny = max(3, round((n / a * b * b) ** (1 / 3)))
        return nx, ny, max(3, round(n / (nx * ny)))

    kind = rng.choice(["tick"] * 6 + ["stepper", "block", "walls", "coupled", "batch", "serve", "grid"])
    disorder = rng.choice([0.01, 0.05, 0.1])
    if kind in ("batch", "serve"):
        top = 131072 if kind == "serve" else 262144
        return dict(kind=kind, scenes=rng.randint(2, 24), lo=rng.randint(2000, 9000), hi=rng.randint(20000, top),
                    mix=rng.randrange(1 << 16), sub=10, ticks=rng.randint(1, 2))
    most = {"tick": 3e6, "stepper": 1e5, "block": 5e5, "walls": 3e5, "coupled": 2e5, "grid": 5e5}[kind]
    nx, ny, nz = dims(log(400, most))
    if kind == "grid":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, s=round(log(0.005, 0.05), 4), bins=rng.choice([1 << 17, 1 << 19]),
                    disorder=disorder)
    ticks = rng.randint(1, 3 if nx * ny * nz < 2e5 else 1)
    if kind == "block":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, s=0.05, sub=4, ticks=ticks, disorder=disorder, u0=0.0)
    s = round(log(0.005, 0.05), 4)
    wide = rng.choice([1.0, 1.0, 1.0, 4.0])  # some tanks far larger than their fluid
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, s=s, tx=round(nx * s * rng.uniform(1.3, 2.5) * wide + 4 * s, 3),
             ty=round(ny * s * rng.uniform(1.2, 1.8) + 6 * s, 3), tz=round(nz * s * rng.uniform(1.0, 1.6) + s, 3),
             sub=rng.choice([4, 10]) if s >= 0.03 else 10, ticks=ticks, disorder=disorder, u0=rng.choice([0.0, 0.3, 0.6]))
    if kind != "walls":
        c["boxes"] = rng.randint(1, 6) if kind in ("stepper", "coupled") else rng.choice([0, 0, 4])
    return c


# ---------------------------------------------------------------- scenes

def _boxes(case, first_id):
    """Boxes on a grid above and beside the fluid, sized by the spacing (sizes and places from the case alone)."""
    n, s = case["boxes"], case["s"]
    if n >= 64:  # dam10m's own boxes
        return scenes.floating_boxes(n, 1002, (1.2, 0.05, 0.05), (2.45, 1.1, 1.15), 0.025, 0.075, first_id, 0.02)
    out = []
    for b in range(n):
        half = (3 * s + 0.4 * s * (b % 3), 2 * s + 0.5 * s * (b % 2), 3 * s)
        place = ((b % 3 + 0.7) / 3.7 * case["tx"], case["ny"] * s + half[1] * (1 + 2.4 * (b // 3)) - s,
                 (0.3 + 0.4 * ((b * 7) % 5) / 4) * case["tz"])
        out.append(scenes.Body(first_id + b, tuple(float(F32(x)) for x in half), tuple(float(F32(x)) for x in place),
                               linvel=(0.1, -0.2, 0.05 * b), angvel=(0.2, 0.0, -0.1 * b)))
    return out


def _slosh(pos, nf, u0, width):
    vel = np.zeros_like(pos)
    if u0:
        vel[:nf, 0] = F32(u0) * np.sin(F32(np.pi) * pos[:nf, 0] / F32(width)).astype(F32)
    return vel


def _scene(case, seed):
    """(spec, bodies): the case's particles, jittered (and set flowing) from the seed."""
    dims, s = (case["nx"], case["ny"], case["nz"]), case["s"]
    fluid = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), dims, s), s, seed, case["disorder"])
    if case["kind"] == "block":
        params = vxl_sph.make_params(smoothing_radius=2.0 * s, substeps=case["sub"])
        params.particle_mass = scenes.lattice_mass(params, s)
        bodies = []
    else:
        params = scenes.baseline_params(s, substeps=case["sub"])
        bodies = [] if case["kind"] == "walls" else scenes.tank_bodies((case["tx"], case["ty"], case["tz"]), 2.0 * s)
        if case.get("boxes"):
            bodies = bodies + _boxes(case, len(bodies))
    spec = scenes.assemble("case", params, fluid, bodies, s, case["ticks"])
    if case.get("u0"):
        spec.vel[:spec.n_fluid] = _slosh(spec.pos, spec.n_fluid, case["u0"], case["tx"])[:spec.n_fluid]
    return spec, bodies


def _tanks(case, seed):
    """Tanks of sizes drawn from case["mix"], their particles from the seed."""
    rng = np.random.Generator(np.random.PCG64(case["mix"]))
    out = []
    for q in range(case["scenes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        kind = "dam" if case["kind"] == "batch" or rng.uniform() < 0.5 else "slosh"
        aspect, fill, s = (float(rng.uniform(*r)) for r in ((0.5, 2.0), (0.2, 0.6), (0.005, 0.02)))
        out.append(scenes.tank_scene(kind, n, s, aspect, fill, seed * 1009 + q, case["ticks"], case["sub"]))
    return out


def _providers(case):
    """Tank faces around [0, t] and a box obstacle beside the fluid."""
    tx, ty, tz, s = case["tx"], case["ty"], case["tz"], case["s"]
    faces = vxl_sph.Faces([(1, 0.0, 1.0), (0, 0.0, 1.0), (0, tx, -1.0), (2, 0.0, 1.0), (2, tz, -1.0)],
                          ((-50.0, -50.0, -50.0), (50.0, 50.0, 50.0)))
    x = case["nx"] * s
    return [faces, scenes.box_obstacle((x + 5 * s, 5 * s, 0.5 * tz), (4 * s, 5 * s, 0.2 * tz))]


def _frames(spec, bodies, ticks):
    """The full particle arrays of each tick of the stepper loop: the boxes (not the walls) move and turn."""
    out = []
    for t in range(ticks):
        moved = []
        for b in bodies:
            if b.linvel != (0.0, 0.0, 0.0):
                a = 0.05 * t
                p = tuple(float(F32(b.pos[k] + b.linvel[k] * t * DT)) for k in range(3))
                b = scenes.Body(b.id, b.half, p, (0.0, float(F32(math.sin(a))), 0.0, float(F32(math.cos(a)))), b.linvel,
                                b.angvel)
            moved.append(b)
        bp, bv, _, spans = scenes.body_particles(moved, spec.spacing, spec.params.smoothing_radius,
                                                 spec.params.boundary_layers, spec.params.rest_density)
        pos, vel = spec.pos.copy(), spec.vel.copy()
        pos[spec.n_fluid:], vel[spec.n_fluid:] = bp, bv
        out.append((pos, vel, [(b, o, i + spec.n_fluid, j + spec.n_fluid) for b, o, i, j in spans]))
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()
    t[...] = a
    return t


def _mass_props(bodies, dynamic):
    """(inverse mass, local inverse inertia) per body: 400 kg/m^3 for the dynamic ones, zeros for the walls."""
    im, ii = np.zeros(len(bodies), F32), np.zeros((len(bodies), 3), F32)
    for q, b in enumerate(bodies):
        if dynamic[q]:
            im[q], ii[q] = scenes.box_mass_props(b.half, 400.0)
    return im, ii


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        s = case["s"]
        pos = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), (case["nx"], case["ny"], case["nz"]), s), s, seed,
                            case["disorder"])
        order = np.random.Generator(np.random.PCG64(seed + 1)).permutation(pos.shape[0])
        info = vxl_sph.GridInfo()
        info.hdr = vxl_sph.header(vxl_sph.GridInfo)
        return dict(case=case, pos=torch.from_numpy(pos[order]).cuda(), info=info, lib=vxl_sph.load(),
                    items=torch.empty(pos.shape[0], dtype=torch.int32, device="cuda"),
                    start=torch.empty(case["bins"] + 1, dtype=torch.int32, device="cuda"))
    if kind in ("batch", "serve"):
        specs = _tanks(case, seed)
        st = dict(case=case, specs=specs)
        if kind == "serve":
            slots, bins = sum(x.n_total for x in specs), len(specs) * (1 << 21)
            st["server"] = vxl_sph.Server((64 << 20) + int(slots * 500 / 0.85) + int(bins * 12 / 0.15))
        else:
            st["batch"] = vxl_sph.Batch(specs)
            st["inputs"] = [(_pinned(x.pos), _pinned(x.vel)) for x in specs]
            st["out"] = _pinned(np.zeros((st["batch"].n_total, 3), F32))
        return st
    spec, bodies = _scene(case, seed)
    st = dict(case=case, spans=spec.spans, pos=_pinned(spec.pos), vel=_pinned(spec.vel), n_fluid=spec.n_fluid)
    st["out"] = (_pinned(np.zeros_like(spec.pos)), _pinned(np.zeros_like(spec.vel)))
    if kind == "stepper":
        st["frames"], st["pmass"] = _frames(spec, bodies, case["ticks"]), spec.pmass
        st["stepper"] = vxl_sph.GpuFluidStepper(spec.params, spec.n_fluid, spec.pos, spec.vel, spec.pmass)
        st["scene"] = st["stepper"].scene
        return st
    st["scene"] = vxl_sph.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    if kind == "walls":
        st["scene"].set_providers(_providers(case))
    if kind == "coupled":
        local, idx = scenes.body_lattice(bodies, spec.spacing, spec.params.smoothing_radius, spec.params.boundary_layers)
        st["scene"].set_body_lattice(local, idx, len(bodies))
        st["scene"].set_spans(spec.spans)
        st["bodies"], st["dynamic"] = bodies, [b.linvel != (0.0, 0.0, 0.0) for b in bodies]
        st["props"] = _mass_props(bodies, st["dynamic"])
    return st


def _reactions(reacts):
    return np.array([[np.concatenate([f, t]) for _, f, t in r] for r in reacts], F32)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "grid":
        pos, items, start, info = st["pos"], st["items"], st["start"], st["info"]
        vp = ctypes.c_void_p
        status = st["lib"].vxl_sph_build_grid_static(vp(pos.data_ptr()), pos.shape[0], 2.0 * case["s"], case["bins"],
                                                     vp(items.data_ptr()), vp(start.data_ptr()), case["bins"] + 1,
                                                     ctypes.byref(info), vp(torch.cuda.current_stream().cuda_stream))
        if status != vxl_sph.OK:
            raise vxl_sph.VxlError(status, "grid build")
        return dict(items=items, start=start[:int(info.total) + 1], dims=list(info.dims))
    if kind == "batch":
        b, reacts = st["batch"], []
        for q, (p, v) in enumerate(st["inputs"]):
            b.write_state(q, p, v)
        for _ in range(case["ticks"] - 1):
            reacts.append(b.step_tick(DT))
        b.step_tick_async(DT)
        b.request_state()
        b.sync()
        reacts.append(b.reactions())
        return dict(pos=b.take_state(st["out"]), react=_reactions(reacts))
    if kind == "serve":
        sv = st["server"]
        ids = [sv.submit(x, case["ticks"]) for x in st["specs"]]
        while True:
            rep = sv.step(DT)
            if not rep.active and not rep.queued:
                break
        return [sv.read(i) for i in ids]
    scene, reacts, more = st["scene"], [], {}
    scene.write_state(st["pos"], st["vel"])
    if kind == "stepper":
        bounds = []
        for pos, vel, spans in st["frames"]:
            st["stepper"].step(DT, st["n_fluid"], pos, vel, st["pmass"], spans)
            reacts.append(st["stepper"].reactions())
            bounds.append(np.stack(st["stepper"].bounds()))
        more["bounds"] = np.stack(bounds)
    elif kind == "coupled":
        scene.set_rigid_bodies(st["bodies"], *st["props"], st["dynamic"])
        for _ in range(case["ticks"]):
            reacts.append(scene.step_coupled(DT, 2, GRAVITY, nspans=len(st["spans"])))
        more["bodies"] = scene.read_rigid_bodies()
    else:
        for _ in range(case["ticks"]):
            reacts.append(scene.step_tick(DT, st["spans"]))
    pos, vel = scene.read_state(out=st["out"])
    if st["spans"]:
        more["react"] = _reactions(reacts)
    return dict(pos=pos, vel=vel, **more)


# ---------------------------------------------------------------- floors

def _counts(case):
    """(fluid, boundary) particles: a wall of thickness 2 s carries a lattice point per s^2 on both faces."""
    nf = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] in ("block", "walls", "grid"):
        return nf, 0
    tx, ty, tz, s = case["tx"], case["ty"], case["tz"], case["s"]
    return nf, 2 * (tx * tz + 2 * ty * tz + 2 * tx * ty) / s ** 2 + case.get("boxes", 0) * (3000 if case["boxes"] >= 64 else 150)


def work(case):
    if case["kind"] == "grid":
        n = _counts(case)[0]
        return dict(bytes=12.0 * n + 4.0 * n + 4.0 * min(case["bins"], n / 8), flops=20.0 * n)
    if case["kind"] in ("batch", "serve"):
        mid = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        nf, nb = case["scenes"] * mid, case["scenes"] * mid * 0.6
    else:
        nf, nb = _counts(case)
    steps = case["sub"] * case["ticks"]
    # a pass: the state in and out; a substep: the fluid's position and velocity read and written, the
    # boundary's read; per pair of the 33 within h = 2 s: a distance and poly6 (12), the force terms (58)
    return dict(bytes=48.0 * (nf + nb) + steps * (48.0 * nf + 24.0 * nb), flops=steps * nf * 33.5 * 70.0)


# ---------------------------------------------------------------- 64-bit rollouts

class _Exact:
    """The WCSPH substep in float64 torch: poly6 density with Akinci boundary terms, Tait pressure, spiky
    pressure force, Monaghan viscosity, XSPH, symplectic Euler with the speed clamp, boundary reactions."""

    def __init__(self, p, pos, vel, pmass, nf, providers=()):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev, self.nf, self.p = dev, nf, p
        self.pos, self.vel, self.m = (torch.from_numpy(np.asarray(a, np.float64)).to(dev) for a in (pos, vel, pmass))
        self.h = float(p.smoothing_radius)
        self.providers = providers
        self.g = torch.tensor(list(p.gravity), dtype=torch.float64, device=dev)

    def planes(self, probe):
        """Contacts of every provider for each fluid particle: (mask, point, normal), in the providers' order."""
        x = self.pos[:self.nf]
        out = []
        for pr in self.providers:
            if isinstance(pr, vxl_sph.Faces):
                for axis, at, sign in pr.faces:
                    n = torch.zeros_like(x)
                    n[:, axis] = sign
                    pt = x.clone()
                    pt[:, axis] = float(F32(at))
                    out.append(((x[:, axis] - float(F32(at))) * sign <= 2 * probe, pt, n))
            else:
                n = torch.tensor([q[0] for q in pr.planes], dtype=torch.float64, device=self.dev)
                d = torch.tensor([float(F32(q[1])) for q in pr.planes], dtype=torch.float64, device=self.dev)
                best, k = (x @ n.T - d).max(1)
                near = best <= probe
                if pr.bounds is not None:
                    lo, hi = (torch.tensor(b, dtype=torch.float64, device=self.dev) for b in pr.bounds)
                    near &= ((x >= lo - self.h) & (x <= hi + self.h)).all(1)
                out.append((near, x - n[k] * best[:, None], n[k]))
        return out

    def edges(self):
        """Every (fluid i, particle j != i) with |pi - pj| <= h: (i, j, d, r2), from cells of side h."""
        x, h, nf = self.pos, self.h, self.nf
        c = ((x - x.min(0).values) / h).floor().long()
        n = c.max(0).values + 1
        key, order = torch.sort((c[:, 0] * n[1] + c[:, 1]) * n[2] + c[:, 2])
        c = c[:nf]
        out = []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                cx, cy = c[:, 0] + dx, c[:, 1] + dy
                ok = (cx >= 0) & (cx < n[0]) & (cy >= 0) & (cy < n[1])
                col = (cx * n[1] + cy) * n[2]
                lo = torch.searchsorted(key, col + (c[:, 2] - 1).clamp(min=0))
                hi = torch.searchsorted(key, col + torch.minimum(c[:, 2] + 1, n[2] - 1), right=True)
                length = torch.where(ok, hi - lo, torch.zeros_like(lo))
                i = torch.repeat_interleave(torch.arange(nf, device=self.dev), length)
                first = torch.cumsum(length, 0) - length
                j = order[torch.arange(i.numel(), device=self.dev) - first[i] + lo[i]]
                d = x[i] - x[j]
                r2 = (d * d).sum(1)
                keep = (r2 <= h * h) & (i != j)
                out.append((i[keep], j[keep], d[keep], r2[keep]))
        return (torch.cat(a) for a in zip(*out))

    def substep(self, dt):
        p, nf, h, m = self.p, self.nf, self.h, self.m
        h2 = h * h
        k6, ks = 315.0 / (64.0 * math.pi * h ** 9), 45.0 / (math.pi * h ** 6)
        i, j, d, r2 = self.edges()
        w = k6 * (h2 - r2) ** 3
        fluid = j < nf
        mass = float(p.particle_mass)
        rho = m * (k6 * h2 ** 3)
        rho[:nf].index_add_(0, i, w * m[j])
        rho.index_add_(0, j[~fluid], w[~fluid] * mass)
        if self.providers:
            x = self.pos[:nf]
            for near, pt, n in self.planes(h):
                sdf = ((x - pt) * n).sum(1)
                e = (near & (sdf > 0) & (sdf < h))[i]
                a, b = i[e], j[e]
                q = self.pos[b]
                g = x[a] - (q - n[a] * (2 * ((q - pt[a]) * n[a]).sum(1))[:, None])
                t = (h2 - (g * g).sum(1)).clamp(min=0)
                rho[:nf].index_add_(0, a, mass * k6 * t ** 3)
        B = float(p.sound_speed) ** 2 * float(p.rest_density) / float(p.gamma_tait)
        pr = B * ((rho / float(p.rest_density)) ** float(p.gamma_tait) - 1)
        if p.tensile_instability_suppression:
            pr = pr.clamp(min=0)
        c = pr / rho ** 2
        r = r2.sqrt()
        spiky = ks * (h - r) ** 2
        dv = self.vel[i] - self.vel[j]
        vdn = -(dv * d).sum(1)
        mu = vdn * h / (r2 + 0.01 * h2)
        alpha = float(p.artificial_viscosity) * float(p.sound_speed)
        visc = torch.where(vdn > 0, alpha * mu / (0.5 * (rho[i] + rho[j])) * spiky, torch.zeros_like(mu))
        f = d * (m[j] * (spiky * (c[i] + c[j]) + visc) / r.clamp(min=1e-9))[:, None]
        acc = self.g.expand(nf, 3).clone().index_add_(0, i, f)
        xs = torch.zeros_like(acc).index_add_(0, i, dv * (-2 * m[j] / (rho[i] + rho[j]) * w)[:, None])
        b = ~fluid
        force = torch.zeros_like(self.pos).index_add_(0, j[b], -mass * f[b])
        u = self.vel[:nf] + acc * dt + xs * float(p.xsph_viscosity)
        top = float(p.max_speed_frac) * h / dt
        u = u * torch.clamp(top / u.norm(dim=1).clamp(min=1e-300), max=1.0)[:, None]
        self.vel[:nf] = u
        self.pos[:nf] += u * dt
        if self.providers:
            self.project()
        return force

    def project(self):
        nf, skin = self.nf, 0.15 * self.h
        x0 = self.pos[:nf].clone()
        nsum, hit, u = torch.zeros_like(x0), torch.zeros(nf, dtype=torch.bool, device=self.dev), self.vel[:nf]
        for near, pt, n in self.planes(skin):  # every contact is taken at the integrated position
            pen = -((x0 - pt) * n).sum(1)
            on = near & (pen > 0)
            self.pos[:nf] += torch.where(on[:, None], n * (pen + skin).clamp(max=self.h)[:, None], torch.zeros_like(n))
            nsum += torch.where(on[:, None], n, torch.zeros_like(n))
            hit |= on
            vn = (u * n).sum(1)
            u -= torch.where((on & (vn < 0))[:, None], n * vn[:, None], torch.zeros_like(n))
        at = hit.nonzero()[:, 0].cpu().numpy()
        x, ns, rmin = self.pos[at].cpu().numpy(), nsum[at].cpu().numpy(), 0.2 * self.h
        length = np.linalg.norm(ns, axis=1)
        for a in range(1, len(at)):  # in reference order, each against the earlier ones as they now stand
            if length[a] <= 1e-9:
                continue
            b = 0
            while b < a:
                r = np.linalg.norm(x[a] - x[b:a], axis=1)
                close = np.nonzero(r < rmin)[0]
                if not close.size:
                    break
                x[a] += ns[a] / length[a] * (rmin - r[close[0]])
                b += int(close[0]) + 1
        self.pos[at] = torch.from_numpy(x).to(self.dev)

    def tick(self, spans):
        """One tick; per span the force and the torque about its origin, averaged over the substeps."""
        sub = int(self.p.substeps)
        total = torch.zeros((len(spans), 6), dtype=torch.float64, device=self.dev)
        for _ in range(sub):
            f = self.substep(float(F32(DT) / F32(sub)))
            for k, (_, origin, a, b) in enumerate(spans):
                arm = self.pos[a:b] - torch.tensor(origin, dtype=torch.float64, device=self.dev)
                total[k, :3] += f[a:b].sum(0)
                total[k, 3:] += torch.linalg.cross(arm, f[a:b]).sum(0)
        return (total / sub).cpu().numpy()


def _turn(q, v):
    t = 2 * np.cross(q[:3], v)
    return v + np.cross(q[:3], t) + q[3] * t


def _integrate(b, force, torque, dt):
    """Two rigid substeps of one dynamic body: gravity, the reaction, semi-implicit Euler."""
    dt = dt / 2
    for _ in range(2):
        b["v"] = b["v"] + (np.array(GRAVITY) + force * b["im"]) * dt
        back = np.array([-b["q"][0], -b["q"][1], -b["q"][2], b["q"][3]])
        b["w"] = b["w"] + _turn(b["q"], _turn(back, torque) * b["ii"]) * dt
        for k, top in (("v", 100.0), ("w", 50.0)):
            b[k] = b[k] * min(1.0, top / max(np.linalg.norm(b[k]), 1e-300))
        b["x"] = b["x"] + b["v"] * dt
        w, q = b["w"], b["q"]
        dq = np.array([w[0] * q[3] + w[1] * q[2] - w[2] * q[1], -w[0] * q[2] + w[1] * q[3] + w[2] * q[0],
                       w[0] * q[1] - w[1] * q[0] + w[2] * q[3], -w[0] * q[0] - w[1] * q[1] - w[2] * q[2]])
        q = q + dq * (0.5 * dt)
        b["q"] = q / np.linalg.norm(q)


def _exact_coupled(case, spec, bodies):
    e = _Exact(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    dynamic = [b.linvel != (0.0, 0.0, 0.0) for b in bodies]
    im, ii = _mass_props(bodies, dynamic)
    local, idx = scenes.body_lattice(bodies, spec.spacing, spec.params.smoothing_radius, spec.params.boundary_layers)
    st = [dict(x=np.array(b.pos, F32).astype(float), q=np.array(b.rot, F32).astype(float),
               v=np.array(b.linvel, F32).astype(float), w=np.array(b.angvel, F32).astype(float), im=float(im[k]),
               ii=ii[k].astype(float)) for k, b in enumerate(bodies)]
    reacts, last = [], np.zeros((len(bodies), 6))
    for _ in range(case["ticks"]):
        pos, vel = np.zeros((len(idx), 3)), np.zeros((len(idx), 3))
        for k, b in enumerate(st):
            if dynamic[k]:
                _integrate(b, last[k, :3], last[k, 3:], DT)
            on = idx == k
            arm = _turn(b["q"], local[on].astype(float))
            pos[on], vel[on] = b["x"] + arm, b["v"] + np.cross(b["w"], arm)
        e.pos[spec.n_fluid:], e.vel[spec.n_fluid:] = torch.from_numpy(pos).to(e.dev), torch.from_numpy(vel).to(e.dev)
        last = e.tick([(k, tuple(b["x"]), i, j) for b, (k, _, i, j) in zip(st, spec.spans)])
        reacts.append(last)
    return dict(pos=e.pos, vel=e.vel, react=np.stack(reacts),
                bodies=np.stack([np.concatenate([b["x"], b["q"], b["v"], b["w"]]) for b in st]))


def _courant(case):
    """c0 dt / h of the 20 m/s constants (of the finest spacing of a set of tanks)."""
    return 20.0 * DT / case["sub"] / (2.0 * case.get("s", 0.005))


def _stiff(case):
    """Past 0.45 the scenes amplify rounding from substep to substep: after more than one tick a velocity in 32 bits
    has no digit in common with one in 64."""
    return case["kind"] != "block" and _courant(case) > 0.45 and case["ticks"] * case["sub"] > 10


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid" or _stiff(case):  # whole numbers; see _stiff
        return None
    # from rest at the finest spacing the velocities of one tick are already as small as their amplified rounding
    lost = kind != "block" and _courant(case) > 1.5 and not case.get("u0")
    if kind in ("batch", "serve"):
        pos, vel, reacts = [], [], []
        for spec in _tanks(case, seed):
            e = _Exact(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
            reacts.append([e.tick(spec.spans) for _ in range(case["ticks"])])
            pos.append(e.pos.cpu().numpy())
            vel.append(None if lost else e.vel.cpu().numpy())
        if kind == "serve":
            return list(zip(pos, vel))
        return dict(pos=np.concatenate(pos), react=np.concatenate(reacts, axis=1))
    spec, bodies = _scene(case, seed)
    if kind == "coupled":
        return _exact_coupled(case, spec, bodies)
    e = _Exact(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid, _providers(case) if kind == "walls" else ())
    reacts, more = [], {}
    if kind == "stepper":
        bounds = []
        for pos, vel, spans in _frames(spec, bodies, case["ticks"]):
            for mine, new in ((e.pos, pos), (e.vel, vel)):
                mine[e.nf:] = torch.from_numpy(new[e.nf:].astype(np.float64)).to(e.dev)
            reacts.append(e.tick(spans))
            bounds.append(torch.stack([e.pos[:e.nf].min(0).values, e.pos[:e.nf].max(0).values]).cpu().numpy())
        more["bounds"] = np.stack(bounds)
    else:
        reacts = [e.tick(spec.spans) for _ in range(case["ticks"])]
    if spec.spans:
        more["react"] = np.stack(reacts)
    return dict(pos=e.pos, vel=None if lost else e.vel, **more)
