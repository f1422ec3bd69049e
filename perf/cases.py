"""The workloads this library's speed is measured on, through its Python
entry points (blaze.device.Simulation, blaze.ensemble.Ensemble,
blaze.calibrate): sphere and polyhedron simulations in reference mode and
with a Verlet list, ensembles with the history laws, the mixed charge of a
turning mill, and a calibration step with gradients.

Beds are in contact and under gravity from the first step.  Box beds are
generated: a face-centred lattice at touching distance with a tenth of its
sites empty and radii spread by 3e-4, so a particle has 6 contacts and
11 candidates in the mean and the counts vary, at a granular temperature of a
few cm/s.  The silo, the hopper, the mill and the mixed charge are the
package's own packings, run until they rest on their walls.  Pass after pass
continues the run, as a program does that reads the state every few steps.
"""
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "softx-d-15-00085_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from blaze import calibrate, device, ensemble as E, synth  # noqa: E402


def listed():
    return [
        # the reference driver's loop on its box world: one call a step, the
        # contact list rebuilt every step, everything bit for bit
        dict(name="call_box_10k", kind="box", n=10_000, steps=1, skin=0.0, spin=True, contracted=False),
        # the same call on the discharging silo at full size
        dict(name="call_silo_1m", kind="silo", n=1_000_000, steps=1, skin=0.0, contracted=False),
        # the silo discharge as it is run for results: Verlet list,
        # contracted law, the state looked at every 16 steps
        dict(name="silo_1m", kind="silo", n=1_000_000, steps=16, skin=0.16, contracted=True),
        # an ordinary box with rotation, bit-exact law, odd size
        dict(name="box_100k", kind="box", n=99_997, steps=16, skin=0.04, spin=True, contracted=False),
        # a coupled host program: state in, one step, state out
        dict(name="roundtrip_200k", kind="roundtrip", n=200_003),
        # ball mill: lifters turned on the device, power tallies on
        dict(name="mill_60k", kind="mill", n=60_000, steps=64, skin=0.05),
        # convex polyhedra (dodecahedra, cubes, hexagonal prisms)
        dict(name="poly_28k", kind="poly", n=28_001, steps=16, skin=0.05),
        # a parameter sweep: many uneven systems at once, persistent stepping
        dict(name="sweep_256", kind="ensemble", systems=256, n_min=2_000, n_max=20_000, steps=32,
             law="linear", graph=2),
        # one small system with the defaults
        dict(name="bed_6k", kind="ensemble", systems=1, n_min=6_001, n_max=6_001, steps=16,
             law="linear", graph=1),
        # Hertz-Mindlin with rolling friction on a 4,096-triangle hopper
        dict(name="hopper_400k", kind="hopper", n=400_000, steps=32),
        # the mill's mixed charge: balls and rocks in a turning mesh of
        # 16,384 triangles
        dict(name="mixed_21k", kind="mixed", balls=20_000, rocks=1_000, steps=32),
        # calibration: forward, loss, gradients of the law constants and of
        # the initial velocities
        dict(name="calibrate_16x4k", kind="adjoint", systems=16, n=4_000, steps=50),
    ]


def draw(rng):
    def size(lo, hi):
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return min(max(v | 1 if rng.random() < 0.7 else v, lo), hi)

    kind = rng.choice(["box", "box", "silo", "roundtrip", "mill", "poly", "ensemble", "ensemble",
                       "hopper", "mixed", "adjoint"])
    if kind == "box":
        ref = rng.random() < 0.4
        return dict(kind=kind, n=size(2_000, 300_000), steps=1 if ref else size(8, 20),
                    skin=0.0 if ref else round(rng.uniform(0.03, 0.06), 3),
                    spin=rng.random() < 0.6, contracted=rng.random() < 0.4)
    if kind == "silo":
        ref = rng.random() < 0.4
        return dict(kind=kind, n=size(60_000, 500_000), steps=1 if ref else size(8, 16),
                    skin=0.0 if ref else round(rng.uniform(0.14, 0.2), 3),
                    contracted=rng.random() < 0.5)
    if kind == "roundtrip":
        return dict(kind=kind, n=size(5_000, 400_000))
    if kind == "mill":
        return dict(kind=kind, n=size(10_000, 100_000), steps=size(16, 64),
                    skin=round(rng.uniform(0.03, 0.06), 3))
    if kind == "poly":
        return dict(kind=kind, n=size(3_000, 60_000), steps=size(4, 16),
                    skin=round(rng.uniform(0.03, 0.06), 3))
    if kind == "ensemble":
        many = rng.random() < 0.5
        lo = size(1_000, 4_000) if many else size(1_000, 100_000)
        return dict(kind=kind, systems=size(8, 256) if many else 1, n_min=lo,
                    n_max=size(lo, 5 * lo) if many else lo, steps=size(4, 32),
                    law=rng.choice(["linear", "hertz"]), graph=rng.choice([1, 2]))
    if kind == "hopper":
        return dict(kind=kind, n=size(50_000, 400_000), steps=size(8, 32))
    if kind == "mixed":
        balls = size(4_000, 30_000)
        return dict(kind=kind, balls=balls, rocks=max(50, balls // rng.randint(15, 40)),
                    steps=size(8, 32))
    return dict(kind=kind, systems=size(2, 16), n=size(500, 4_000), steps=size(24, 50))


# ------------------------------------------------------------------ inputs
R = 0.2                    # box beds: mean radius, cm
SPREAD = 3e-4              # relative spread of the radii
HEAT = 10.0                # standard deviation of the velocities, cm/s
DT = 5e-6


def _lattice(n):
    """n random sites of 1.1 n lowest ones of a face-centred lattice at
    touching distance in a box of about equal sides, and the box: (sites
    chooser input, L, H)."""
    s = 2.0 * R / math.sqrt(2.0)                    # x + y + z even, times s
    want = int(math.ceil(1.1 * n))
    m = max(2, int(round((2.0 * want) ** (1.0 / 3.0))))
    k = int(math.ceil(2.0 * want / (m * m))) + 1
    L = (m - 1) * s + 2.0 * R
    H = (1.5 * k) * s + 4.0 * R
    return s, m, k, want, L, H


def _bed(n, gen):
    """(positions, radii, velocities, spins) of a generated box bed, float32
    on the GPU, in random order; and its box L, H."""
    dev = "cuda"
    s, m, k, want, L, H = _lattice(n)
    idx = torch.arange(m * m * k, device=dev)
    x, y, z = idx % m, (idx // m) % m, idx // (m * m)
    keep = ((x + y + z) % 2 == 0).nonzero().flatten()[:want]
    keep = keep[torch.randperm(len(keep), device=dev, generator=gen)[:n]]
    pos = torch.stack([x[keep], y[keep], z[keep]], 1).double() * s + R
    f32 = dict(device=dev, generator=gen)
    pos = (pos + 1e-4 * R * torch.randn(n, 3, **f32).double()).float()
    vel = HEAT * torch.randn(n, 3, **f32)
    spin = HEAT / R * torch.randn(n, 3, **f32)
    return pos, vel, spin, L, H


def _radii(n, gen, bins=0):
    u = torch.rand(n, device="cuda", generator=gen).double() * 2.0 - 1.0
    if bins:
        u = ((u + 1.0) / 2.0 * bins).floor().clamp(max=bins - 1) / (bins - 1) * 2.0 - 1.0
    return (R * (1.0 + SPREAD * u)).float()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _np(t):
    return t.cpu().numpy()


@functools.lru_cache(maxsize=2)
def _box_project(n, spin):
    """The reference project of a box bed: six radius bins, six quads."""
    _, _, _, _, L, H = _lattice(n)
    bins = np.unique(_np(_radii(10_000, _gen(0), bins=6)))
    S = synth.box_system(n, L, H, 2.0 * float(bins.max()), 0, density=2500e-6, kn=1e5,
                         restitution=0.5, mu=0.4)
    with tempfile.TemporaryDirectory() as d:
        P, _ = synth.box_system_project(d, "Box", S, L, H, bins, 2500.0, dt=DT)
    P.sim_info.Num_Particles = n
    P.sim_info.Rotation = bool(spin)
    return P, bins


def _box_state(n, seed, spin):
    g = _gen(seed)
    P, bins = _box_project(n, spin)
    rad = _np(_radii(n, g, bins=6))
    pos, vel, avel, _, _ = _bed(n, g)
    return P, dict(pos=_np(pos), vel=_np(vel), avel=_np(avel if spin else 0.0 * avel),
                   type=np.searchsorted(bins, rad).astype(np.uint32),
                   pid=np.arange(n, dtype=np.int32))


def _run_to(sim, st, steps):
    sim.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"])
    sim.step(steps)
    out = sim.state()
    order = np.argsort(out["pid"])
    return {k: np.ascontiguousarray(out[k][order]) for k in ("pos", "vel", "avel", "type", "pid")}


@functools.lru_cache(maxsize=4)
def _silo(n):
    """The discharge silo's project and its bed at rest on the closed hatch
    (48,000 steps)."""
    with tempfile.TemporaryDirectory() as d:
        P, st = synth.silo_project(d, n=n)
    sim = device.Simulation(P, skin=0.16, use_graph=1)
    out = _run_to(sim, st, 48_000)
    sim.close()
    return P, out


@functools.lru_cache(maxsize=4)
def _mill(n):
    """The mill's project and its charge as it reaches the standing drum and
    lifters (44,000 steps)."""
    with tempfile.TemporaryDirectory() as d:
        P, st = synth.mill_project(d, n=n)
    sim = device.Simulation(P, skin=0.05, use_graph=1)
    out = _run_to(sim, st, 44_000)
    sim.close()
    return P, out


@functools.lru_cache(maxsize=4)
def _poly(n):
    """The box of polyhedra, fallen together for 16,000 steps."""
    with tempfile.TemporaryDirectory() as d:
        P, st = synth.poly_box_project(d, n=n, spacing=0.99, jitter=0.005)
    sim = device.Simulation(P, skin=0.05, use_graph=1)
    sim.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"], quat=st["quat"])
    sim.step(16_000)
    out = sim.state()
    sim.close()
    order = np.argsort(out["pid"])
    return P, {k: np.ascontiguousarray(out[k][order])
               for k in ("pos", "vel", "avel", "type", "pid", "quat")}


def _ens_settled(ens, pos, rad, steps, vel=None):
    ens.set_state(pos, rad, vel)
    ens.step(steps)
    out = ens.state()
    order = np.argsort(out["pid"])
    return {k: np.ascontiguousarray(out[k][order]) for k in ("pos", "radius", "vel", "avel")}


HOPPER = dict(law=E.LAW_HERTZ_MINDLIN, dt=5e-6, skin=0.04)
MIXED = dict(law=E.LAW_LINEAR, dt=2e-6, skin=0.04)


@functools.lru_cache(maxsize=4)
def _hopper(n):
    systems, walls, pos, rad = synth.silo_full_ensemble(n=n)
    ens = E.Ensemble(systems, walls, **HOPPER)
    st = _ens_settled(ens, pos, rad, 30_000)
    ens.close()
    return systems, walls, st


@functools.lru_cache(maxsize=4)
def _mixed(balls, rocks):
    """The mixed charge's systems, walls and shapes, and the charge at rest in
    the standing drum."""
    systems, walls, pos, rad, shapes, shape_of, quat = synth.mill_mixed_ensemble(
        n_spheres=balls, n_rocks=rocks)
    still = [E.System.from_buffer_copy(bytes(s)) for s in systems]
    for s in still:
        s.rot_omega = 0.0
    ens = E.Ensemble(still, walls, **MIXED)
    ens.set_state(pos, rad)
    ens.set_polyhedra(shapes, shape_of, quat)
    ens.step(60_000)
    out, q = ens.state(), ens.orientations()
    ens.close()
    order = np.argsort(out["pid"])
    st = {k: np.ascontiguousarray(out[k][order]) for k in ("pos", "radius", "vel", "avel")}
    return systems, walls, st, shapes, shape_of, q[order]


def _ensemble_inputs(case, seed):
    """Systems, walls and concatenated arrays of box beds of uneven sizes."""
    g = _gen(seed)
    counts = synth.batched_counts(case["systems"], case["n_min"], case["n_max"])
    rng = np.random.default_rng(7)
    systems, walls, arrs = [], [], []
    cell = 2.0 * R * (1.0 + SPREAD) + 0.04
    for n in counts:
        n = int(n)
        pos, vel, avel, L, H = _bed(n, g)
        mu, e = float(rng.uniform(0.2, 0.8)), float(rng.uniform(0.3, 0.9))
        systems.append(synth.box_system(n, L, H, cell, len(walls), density=2500e-6, kn=1e5,
                                        youngs=1e5, restitution=e, mu=mu,
                                        mu_roll=0.01 if case["law"] == "hertz" else 0.0))
        walls += synth.box_walls(L, H)
        arrs.append((pos, _radii(n, g), vel, avel))
    return systems, walls, [_np(torch.cat(a)) for a in zip(*arrs)]


def _ensemble_options(case):
    law = E.LAW_LINEAR if case["law"] == "linear" else E.LAW_HERTZ_MINDLIN
    return dict(law=law, dt=DT, skin=0.03, use_graph=case["graph"])


def _adjoint_inputs(case, seed):
    systems, walls, pos, rad = _calibration(case["systems"], case["n"])
    n = len(pos)
    rng = np.random.default_rng(int(seed))
    v0 = calibrate.initial_velocity(n, seed=int(seed) % (1 << 30))
    w = rng.normal(size=(2, n, 3))
    params = np.stack([np.array([1e5, 0.5, 0.4, 0.4]) * rng.uniform(0.8, 1.2, 4)
                       for _ in systems])
    return systems, walls, pos, rad, params, v0, w


@functools.lru_cache(maxsize=2)
def _calibration(nsys, n):
    return calibrate.calibration_ensemble(nsys=nsys, n=n)


def _heat(st, seed, scale):
    """The settled bed's velocities with a seeded part on top."""
    g = _gen(seed)
    return st["vel"] + _np(scale * torch.randn(*st["vel"].shape, device="cuda", generator=g))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("box", "roundtrip"):
        spin = case.get("spin", True)
        P, st = _box_state(case["n"], seed, spin)
        sim = device.Simulation(P, skin=case.get("skin", 0.0), use_graph=1,
                                fast_law=int(case.get("contracted", False)))
        sim.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"])
        if kind == "roundtrip":
            return dict(kind=kind, sim=sim, st=st)
        sim.prepare_graphs()
        return dict(kind=kind, sim=sim, steps=case["steps"], views={})
    if kind == "silo":
        P, st = _silo(case["n"])
        sim = device.Simulation(P, skin=case["skin"], use_graph=1,
                                fast_law=int(case["contracted"]))
        sim.set_state(st["pos"], _heat(st, seed, 2.0), st["avel"], st["type"], st["pid"])
        sim.open_hatch()
        sim.prepare_graphs()
        return dict(kind=kind, sim=sim, steps=case["steps"], views={})
    if kind == "mill":
        P, st = _mill(case["n"])
        sim = device.Simulation(P, skin=case["skin"], use_graph=1)
        sim.set_cylinder_rotation(True)
        sim.set_state(st["pos"], _heat(st, seed, 5.0), st["avel"], st["type"], st["pid"])
        axis = float(P.wobj[0].cyl_geo.radius)
        sim.set_dobj_rotation(axis, axis, float(P.mill.RadPerStep))
        sim.prepare_graphs()
        return dict(kind=kind, sim=sim, steps=case["steps"], views={})
    if kind == "poly":
        P, st = _poly(case["n"])
        sim = device.Simulation(P, skin=case["skin"], use_graph=1)
        sim.set_state(st["pos"], _heat(st, seed, 5.0), st["avel"], st["type"], st["pid"],
                      quat=st["quat"])
        sim.prepare_graphs()
        return dict(kind=kind, sim=sim, steps=case["steps"], views={})
    if kind == "ensemble":
        systems, walls, (pos, rad, vel, avel) = _ensemble_inputs(case, seed)
        ens = E.Ensemble(systems, walls, **_ensemble_options(case))
        ens.set_state(pos, rad, vel, avel)
        return dict(kind=kind, sim=ens, steps=case["steps"], views={})
    if kind == "hopper":
        systems, walls, st = _hopper(case["n"])
        ens = E.Ensemble(systems, walls, **HOPPER)
        ens.set_state(st["pos"], st["radius"], _heat(st, seed, 2.0), st["avel"])
        return dict(kind=kind, sim=ens, steps=case["steps"], views={})
    if kind == "mixed":
        systems, walls, st, shapes, shape_of, quat = _mixed(case["balls"], case["rocks"])
        ens = E.Ensemble(systems, walls, **MIXED)
        ens.set_state(st["pos"], st["radius"], _heat(st, seed, 5.0), st["avel"])
        ens.set_polyhedra(shapes, shape_of, quat)
        return dict(kind=kind, sim=ens, steps=case["steps"], views={})
    systems, walls, pos, rad, params, v0, w = _adjoint_inputs(case, seed)
    runner = calibrate.Runner(systems, walls, pos, rad, case["steps"], segment=25, dt=1e-5,
                              tape_bytes=2 << 30)
    return dict(kind=kind, runner=runner, params=torch.from_numpy(params),
                v0=torch.from_numpy(v0), w=torch.from_numpy(w))


# -------------------------------------------------------------------- a pass
class _Shared:
    """Device memory of a simulation as torch sees it; keeps the simulation."""

    def __init__(self, sim, ptr):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (sim.n, 4), "typestr": "<f4",
                                         "data": (int(ptr), False), "version": 2}


def _views(s):
    """The current state on the device: positions with radii, velocities,
    spins (memory order)."""
    sim = s["sim"]
    ptrs = sim.device_state()[:3]
    v = s["views"].get(ptrs[0])
    if v is None:
        v = [torch.as_tensor(_Shared(sim, p), device="cuda") for p in ptrs]
        v = s["views"][ptrs[0]] = (v[0], v[1][:, :3], v[2][:, :3])
    return v


def run(state):
    s = state
    kind = s["kind"]
    if kind == "roundtrip":
        st, sim = s["st"], s["sim"]
        sim.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"])
        sim.step(1)
        out = sim.state()
        return [out["pos"], out["vel"], out["avel"], out["pid"]]
    if kind == "adjoint":
        params = s["params"].clone().requires_grad_(True)
        v0 = s["v0"].clone().requires_grad_(True)
        pos, vel = calibrate.EnsembleRun.apply(params, v0, s["runner"])
        loss = (s["w"][0] * pos).sum() + 1e-3 * (s["w"][1] * vel).sum()
        loss.backward()
        return [pos.detach(), vel.detach(), params.grad, v0.grad]
    s["sim"].step(s["steps"])
    out = list(_views(s))
    if kind == "mill":
        out.append(s["sim"].energy())
    return out


def _count(case):
    kind = case["kind"]
    if kind == "ensemble":
        return int(synth.batched_counts(case["systems"], case["n_min"], case["n_max"]).sum())
    if kind == "mixed":
        return case["balls"] + case["rocks"]
    if kind == "adjoint":
        return case["systems"] * case["n"]
    return case["n"]


def work(case):
    """A particle-step reads and writes the state once (96 bytes; with
    orientations 128) and evaluates 6 contacts of about 100 operations; a
    history contact also reads and writes its 12-byte spring.  A polyhedron's
    contacts are some 12 separating-axis tests of a thousand operations."""
    kind, n, steps = case["kind"], _count(case), case.get("steps", 1)
    bytes_, flops = 96.0 * n * steps, 600.0 * n * steps
    if kind == "poly":
        bytes_, flops = 128.0 * n * steps, 12_000.0 * n * steps
    elif kind in ("ensemble", "hopper"):
        bytes_ += 144.0 * n * steps
    elif kind == "mixed":
        bytes_ += (144.0 * case["balls"] + 600.0 * case["rocks"]) * steps
        flops += 20_000.0 * case["rocks"] * steps
    elif kind == "adjoint":
        bytes_, flops = 4.0 * (96.0 + 72.0) * n * steps, 4.0 * 600.0 * n * steps
    elif kind == "roundtrip":
        bytes_ += 88.0 * n
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """The uncontracted sphere and polyhedron paths promise the reference's
    numbers bit for bit.  Elsewhere a stiff contact amplifies the rounding of
    the overlaps within a pass: against 64 bits the velocities are 0.004 off
    after 16 contracted silo steps, the spins 0.016 after 32 ensemble steps, the
    gradients 0.024 after 50; another correct rounding is about as far off."""
    if case["kind"] in ("mill", "poly", "roundtrip") or not case.get("contracted", True):
        return "exact"
    return {"rel": 0.015} if case["kind"] in ("box", "silo") else {"rel": 0.03}


# ------------------------------------------------- the same in 64 bits
def _f64(a):
    return torch.as_tensor(np.asarray(a), device="cuda").double()


def _pairs(pos, rad, cut, block=None):
    """Index pairs i < j with |xi - xj| < ri + rj + cut (and the same entry
    of `block`), by cells of the largest reach."""
    n = len(pos)
    reach = float(2.0 * rad.max() + cut)
    lo = pos.min(0).values - 1e-9
    c = ((pos - lo) / reach).floor().long()
    nc = c.max(0).values + 3
    b = torch.zeros(n, dtype=torch.long, device=pos.device) if block is None else block
    key = ((b * nc[2] + c[:, 2] + 1) * nc[1] + c[:, 1] + 1) * nc[0] + c[:, 0] + 1
    order = key.argsort()
    ks = key[order]
    got = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key + (dz * nc[1] + dy) * nc[0] + dx
                if (dz, dy, dx) < (0, 0, 0):
                    continue
                s = torch.searchsorted(ks, k)
                e = torch.searchsorted(ks, k, right=True)
                live = torch.arange(n, device=pos.device)
                t = 0
                while True:
                    live = live[(e - s)[live] > t]
                    if not len(live):
                        break
                    j = order[s[live] + t]
                    ok = (pos[live] - pos[j]).norm(dim=1) < rad[live] + rad[j] + cut
                    ok &= b[live] == b[j]
                    if (dz, dy, dx) == (0, 0, 0):
                        ok &= live < j
                    got.append(torch.stack([live[ok], j[ok]]))
                    t += 1
    p = torch.cat(got, 1)
    return p[0], p[1]


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _faces(P, n_w):
    """(normal, centroid, vertices, area, tolerance) of every planar face."""
    out = []
    v3 = lambda a: np.array([a.x, a.y, a.z], np.float32)  # noqa: E731
    for o in range(n_w):
        W = P.wobj[o]
        for q in range(W.num_surfaces):
            F = W.surfaces[q]
            vs = np.stack([v3(W.vertex[F.vertex_Order[k]]) for k in range(F.num_vertex)])
            out.append((_f64(v3(F.normal)), _f64(v3(F.centroid)), _f64(vs), F.area, F.Tol))
    return out


def _reference_run(P, n_w, st, steps):
    """The reference's sphere step with planar faces, in 64 bits."""
    pos, vel, avel = _f64(st["pos"]), _f64(st["vel"]), _f64(st["avel"])
    ty = torch.as_tensor(st["type"].astype(np.int64), device="cuda")
    nt, si = P.n_p, P.sim_info
    ob = [P.pobj[t] for t in range(nt)]
    col = lambda f: _f64([np.float32(f(o)) for o in ob])[ty][:, None]  # noqa: E731
    rad, mass = col(lambda o: o.radius), col(lambda o: o.mass)
    iinv = col(lambda o: o.InertiaT[0])
    s_kn, s_cn = col(lambda o: o.surface_Kn), col(lambda o: o.surface_Cn)
    s_mu = col(lambda o: o.surface_Fric_static)
    kn, cn, mu = (_f64([[np.float32(getattr(a.PP[b], f)) for b in range(nt)] for a in ob])
                  for f in ("Kn", "Cn", "Fric_kinetic"))
    dt = float(si.InitalDelta_t)
    g = _f64([si.Force_Field.x, si.Force_Field.y, si.Force_Field.z])
    spin = bool(si.Rotation)
    i, j = _pairs(pos, rad[:, 0], float(2.0 * vel.norm(dim=1).max()) * dt * steps + 0.02)
    k1, c1, m1 = kn[ty[i], ty[j]][:, None], cn[ty[i], ty[j]][:, None], mu[ty[i], ty[j]][:, None]
    faces = _faces(P, n_w)
    for _ in range(steps):
        f, tq = g * mass, torch.zeros_like(pos)
        rel = pos[i] - pos[j]
        d = rel.norm(dim=1, keepdim=True)
        on = (d - (rad[i] + rad[j]) < 0).flatten().nonzero().flatten()
        a, b, d, rel = i[on], j[on], d[on], rel[on]
        nrm, pen = rel / d, (d - (rad[a] + rad[b])).abs() + 1e-5
        rv = vel[a] - vel[b]
        ra, rb = -nrm * rad[a], nrm * rad[b]
        F = k1[on] * pen * nrm - c1[on] * _dot(rv, nrm) * nrm
        dv = vel[a] + _cross(avel[a], ra) - vel[b] - _cross(avel[b], rb)
        vt = dv - _dot(dv, nrm) * nrm
        vr = rv.norm(dim=1, keepdim=True)
        F = F - (0.5 * (mass[a] + mass[b]) / dt * 0.05) * m1[on] / torch.where(vr > 0, vr, 1.0) * vt
        f.index_add_(0, a, F)
        f.index_add_(0, b, -F)
        tq.index_add_(0, a, _cross(ra, F))
        tq.index_add_(0, b, _cross(-rb, F))
        for nf, cf, vs, area, tol in faces:
            dis = ((pos - rad * nf - cf) @ nf)
            w = ((dis < 0) & (dis > -rad[:, 0])).nonzero().flatten()
            if not len(w):
                continue
            pt = pos[w] - rad[w] * nf
            pen = dis[w].abs()[:, None]
            q = pt + nf * pen
            e = vs[None] - q[:, None]
            ar = 0.5 * _cross(e, e.roll(-1, 1)).norm(dim=2).sum(1)
            ok = (ar - area).abs() / area * 100.0 <= tol
            w, pt, pen = w[ok], pt[ok], pen[ok]
            v = vel[w]
            vn = _dot(v, nf) * nf
            F = s_kn[w] * pen * nf - s_cn[w] * vn
            F = torch.where(_dot(F, nf) < 0, s_kn[w] * pen * nf, F)
            lever = pt - pos[w]
            vt = v - vn + (_cross(avel[w], lever) if spin else 0.0)
            vm = v.norm(dim=1, keepdim=True)
            F = F - 0.05 * mass[w] / dt * s_mu[w] / torch.where(vm > 0, vm, 1.0) * vt
            f.index_add_(0, w, F)
            tq.index_add_(0, w, _cross(lever, F))
        vel = vel + f / mass * dt
        pos = pos + vel * dt
        if spin:
            avel = avel + iinv * tq * dt
    return pos, rad, vel, avel


def _sorted_order(P, st, skin):
    """Memory order after the re-sort the first step makes: stable by cell,
    cells of the project or, with a skin, of at least 2 r_max + skin."""
    si = P.sim_info
    f = np.float32
    cell = [f(si.cellSize.x), f(si.cellSize.y), f(si.cellSize.z)]
    nc = [si.num_NNCells.x, si.num_NNCells.y, si.num_NNCells.z]
    if skin > 0:
        need = f(2.0) * max(f(P.pobj[t].radius) for t in range(P.n_p)) + f(skin)
        for a in range(3):
            if cell[a] < need:
                nc[a] = max(1, int(math.ceil(float(nc[a]) * float(cell[a]) / float(need))))
                cell[a] = need
    org = [f(si.worldOrigin.x), f(si.worldOrigin.y), f(si.worldOrigin.z)]
    x, y, z = (np.floor((st["pos"][:, a] - org[a]) / cell[a]).astype(np.int64) for a in range(3))
    return np.argsort(x + z * nc[2] + y * nc[0] * nc[2], kind="stable")


def _ensemble_run(systems, walls, pos, rad, vel, avel, steps, law, dt, consts=None):
    """The history laws in box systems of planes, in 64 bits.  consts: per
    system (kn, kt, 2 beta, mu, mu_wall) tensors (gradients flow through)."""
    n = len(pos)
    cnt = [s.n for s in systems]
    sy = torch.repeat_interleave(torch.arange(len(cnt), device="cuda"),
                                 torch.tensor(cnt, device="cuda"))
    per = lambda f: _f64([f(s) for s in systems])  # noqa: E731
    if consts is None:
        le = np.log([float(np.float32(s.restitution)) for s in systems])
        beta = _f64(-le / np.sqrt(le * le + np.pi ** 2))
        consts = (per(lambda s: s.kn), per(lambda s: s.kn) * per(lambda s: s.kt_ratio), 2.0 * beta,
                  per(lambda s: s.mu), per(lambda s: s.mu_wall))
    kn, kt, b2, mu, muw = consts
    es = per(lambda s: s.youngs) / (2.0 * (1.0 - per(lambda s: s.poisson) ** 2))
    gs = per(lambda s: s.youngs) / (4.0 * (2.0 - per(lambda s: s.poisson)) *
                                    (1.0 + per(lambda s: s.poisson)))
    mur = per(lambda s: s.mu_roll)
    g = torch.stack([_f64(list(s.gravity)) for s in systems])[sy]
    r = rad[:, None]
    m = (per(lambda s: s.density) * 4.0 / 3.0 * math.pi)[sy][:, None] * r ** 3
    inertia = 0.4 * m * r * r
    vmax = float(vel.norm(dim=1).max())
    i, j = _pairs(pos.detach(), rad, 2.0 * vmax * dt * steps + 0.1 * R, sy)
    planes = [torch.stack([_f64(list(walls[s.wall0 + q].p)[:4]) for s in systems])[sy]
              for q in range(6)]
    xi = torch.zeros(len(i), 3, dtype=torch.float64, device="cuda")
    xw = [torch.zeros(n, 3, dtype=torch.float64, device="cuda") for _ in planes]

    def contact(s, muc, nrm, delta, rs, ms, vrel, vct, wrel, x):
        c = lambda t: t[s][:, None]  # noqa: E731
        if law == "linear":
            kne, kte = c(kn), c(kt)
            cn, ct = c(b2) * (ms * c(kn)).sqrt(), c(b2) * (ms * c(kt)).sqrt()
        else:
            sq = (rs * delta).sqrt()
            sn, kte = 2.0 * c(es) * sq, 8.0 * c(gs) * sq
            kne, bh = 2.0 / 3.0 * sn, math.sqrt(5.0 / 6.0) * c(b2)
            cn, ct = bh * (sn * ms).sqrt(), bh * (kte * ms).sqrt()
        fn = kne * delta - cn * _dot(vrel, nrm)
        fc = fn.clamp(min=0.0)
        vt = vct - _dot(vct, nrm) * nrm
        m0 = _dot(x, x)
        x1 = x - _dot(x, nrm) * nrm
        m1 = _dot(x1, x1)
        ok = m1 > 0
        x = torch.where(ok, x1 * (torch.where(ok, m0, 1.0) / torch.where(ok, m1, 1.0)).sqrt(), x1)
        x = x + vt * dt
        ft = -kte * x - ct * vt
        f2 = _dot(ft, ft)
        cap = c(muc) * fc
        slip = f2 > cap * cap
        fs = ft * cap / torch.where(slip, f2, 1.0).sqrt()
        ft = torch.where(slip, fs, ft)
        x = torch.where(slip, -(ft + vt * ct) / kte, x)
        w2 = _dot(wrel, wrel)
        roll = -c(mur) * fc * rs / torch.where(w2 > 0, w2, 1.0).sqrt() * wrel
        return nrm * fn + ft, roll, x

    for _ in range(steps):
        f, tq = torch.zeros_like(pos), torch.zeros_like(pos)
        rel = pos[i] - pos[j]
        d = rel.norm(dim=1, keepdim=True)
        dl = r[i] + r[j] - d
        on = (dl > 0).flatten().nonzero().flatten()
        a, b, nrm = i[on], j[on], (rel / d)[on]
        ca, cb = -nrm * r[a], nrm * r[b]
        F, T, x = contact(sy[a], mu, nrm, dl[on], r[a] * r[b] / (r[a] + r[b]),
                          m[a] * m[b] / (m[a] + m[b]), vel[a] - vel[b],
                          vel[a] + _cross(avel[a], ca) - vel[b] - _cross(avel[b], cb),
                          avel[a] - avel[b], xi[on])
        xi = torch.zeros_like(xi).index_put((on,), x)
        f = f.index_add(0, a, F).index_add(0, b, -F)
        tq = tq.index_add(0, a, _cross(ca, F) + T).index_add(0, b, _cross(-cb, F) - T)
        for q, pl in enumerate(planes):
            dl = r + pl[:, 3:] - _dot(pl[:, :3], pos)
            on = (dl > 0).flatten().nonzero().flatten()
            nrm = pl[on, :3]
            c1 = -nrm * r[on]
            F, T, x = contact(sy[on], muw, nrm, dl[on], r[on], m[on], vel[on],
                              vel[on] + _cross(avel[on], c1), avel[on], xw[q][on])
            xw[q] = torch.zeros_like(xw[q]).index_put((on,), x)
            f = f.index_add(0, on, F)
            tq = tq.index_add(0, on, _cross(c1, F) + T)
        vel = vel + (f / m + g) * dt
        pos = pos + vel * dt
        avel = avel + tq / inertia * dt
    return pos, vel, avel


def _ensemble_order(systems, pos):
    off, k, keys = 0, 0, []
    for s in systems:
        p = pos[k:k + s.n]
        k += s.n
        c = np.floor((p - np.array(list(s.origin), np.float32)) / np.float32(s.cell)).astype(np.int64)
        nx, ny, nz = list(s.ncells)
        keys.append(off + c[:, 0] + nx * (c[:, 1] + ny * c[:, 2]))
        off += nx * ny * nz
    return np.argsort(np.concatenate(keys), kind="stable")


def exact(case, seed):
    kind = case["kind"]
    # lifters, hulls and triangle meshes: a plain 64-bit form would run for
    # minutes
    if kind in ("mill", "poly", "hopper", "mixed"):
        return None
    if kind in ("box", "silo", "roundtrip"):
        if kind == "silo":
            P, st = _silo(case["n"])
            st = dict(st, vel=_heat(st, seed, 2.0))
            n_w = P.n_w - 1                       # the hatch is open
        else:
            P, st = _box_state(case["n"], seed, case.get("spin", True))
            n_w = P.n_w
        order = torch.as_tensor(_sorted_order(P, st, case.get("skin", 0.0)), device="cuda")
        pos, rad, vel, avel = (t[order] for t in _reference_run(P, n_w, st, case.get("steps", 1)))
        if kind == "roundtrip":
            return [pos, vel, avel, order.int()]
        return [torch.cat([pos, rad], 1), vel, avel]
    if kind == "ensemble":
        systems, walls, arrs = _ensemble_inputs(case, seed)
        order = torch.as_tensor(_ensemble_order(systems, arrs[0]), device="cuda")
        pos, rad, vel, avel = (_f64(a) for a in arrs)
        pos, vel, avel = _ensemble_run(systems, walls, pos, rad, vel, avel, case["steps"],
                                       case["law"], DT)
        return [torch.cat([pos, rad[:, None]], 1)[order], vel[order], avel[order]]
    systems, walls, pos, rad, params, v0, w = _adjoint_inputs(case, seed)
    p = _f64(params).requires_grad_(True)
    # the run takes the parameters and velocities as float32
    p32 = p + (_f64(params.astype(np.float32)) - _f64(params))
    v = _f64(v0).requires_grad_(True)
    v32 = v + (_f64(v0.astype(np.float32)) - _f64(v0))
    le = torch.log(p32[:, 1])
    ratio = _f64([s.kt_ratio for s in systems])
    consts = (p32[:, 0], p32[:, 0] * ratio, -2.0 * le / (le * le + math.pi ** 2).sqrt(), p32[:, 2],
              p32[:, 3])
    x, u, _ = _ensemble_run(systems, walls, _f64(pos), _f64(rad), v32, torch.zeros_like(v32),
                            case["steps"], "linear", 1e-5, consts)
    wt = _f64(w)
    ((wt[0] * x).sum() + 1e-3 * (wt[1] * u).sum()).backward()
    return [x.detach(), u.detach(), p.grad, v.grad]
