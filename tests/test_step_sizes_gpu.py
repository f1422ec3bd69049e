"""The step kernels at the sizes where their launch changes: how many particles
a warp takes (it shares its contacts among its lanes), rounds or IF nodes in
graph stepping, persistent stepping's resident grid, the block sums of the
energy tallies and the lifters' turn in the step's last block, and the windows
of candidate triangles of a polyhedron.  Spheres against the FP32 restatements
bit for bit (the energy sums are FP64 sums of at most some 5e5 terms of one
sign in another order: within 5e5 x 2^-53 < 1e-10), stepping modes against each other bit for bit."""
import math

import numpy as np
import pytest

from bindings import EnsRestated, Restated
from blaze import device, synth
from blaze import ensemble as E
from blaze import types as T

pytestmark = pytest.mark.gpu


def lattice(n, pitch, origin, seed):
    """The first n sites of a cubic lattice, random order, jittered; and its side."""
    rng = np.random.default_rng(seed)
    m = int(math.ceil(n ** (1.0 / 3.0)))
    g = np.arange(m ** 3)[:n]
    p = np.stack([g % m, g // m % m, g // (m * m)], 1) * pitch + origin
    p = p + rng.uniform(-1e-4, 1e-4, p.shape)
    return p[rng.permutation(n)].astype(np.float32), rng, m * pitch


# the tallies' block sums: one size above a block, many blocks, and without shared contacts
@pytest.mark.parametrize("n,energy", [(n, False) for n in (1, 33, 257, 14208, 14209, 28417, 56832, 56833)] +
                         [(n, True) for n in (257, 14209, 56833, 100000, 100001)])
def test_sphere_step_sizes(tmp_path, n, energy):
    r = 0.1
    P, _ = synth.box_project(str(tmp_path), n_side=(2, 2, 2), radius=r)
    P.sim_info.Num_Particles = n
    P.sim_info.EnergyCalc = energy
    pos, rng, _ = lattice(n, 0.1995, 0.0995, n)       # touching the walls and each other
    vel = rng.normal(scale=10.0, size=(n, 3)).astype(np.float32)
    avel = rng.normal(scale=30.0, size=(n, 3)).astype(np.float32)
    ty, pid = np.zeros(n, np.uint32), np.arange(n, dtype=np.int32)
    ref = Restated("f32").init(P.sim_info, P.wobj, P.n_w, P.pobj, P.n_p, P.dobj, P.n_d)
    ref.set_state(pos, vel, avel, ty, pid)
    sims = [device.Simulation(P, use_graph=g) for g in (0, 1)]
    for s in sims:
        s.set_state(pos, vel, avel, ty, pid)
        s.step(1)
        s.step(2)
    ref.step(3)
    want = ref.state()
    for s in sims:
        got = s.state()
        assert got["status"] == 0
        for k in ("pos", "vel", "avel"):
            np.testing.assert_array_equal(got[k].astype(np.float64), want[k], err_msg=k)
        np.testing.assert_array_equal(got["pid"], want["pid"])
        if energy:
            e, w = s.energy(), np.asarray(ref.energy(), np.float64)
            assert e[0] > 0 and e[2] > 0
            np.testing.assert_allclose(e, w, rtol=1e-10)
    np.testing.assert_array_equal(sims[0].energy(), sims[1].energy())
    for s in sims:
        s.close()


def ens_box(n):
    """One box system in contact, hot enough to re-sort every few steps."""
    r = 0.2
    pos, rng, side = lattice(n, 0.4 - 2e-4, 0.2, n)
    L, H = side + 0.02, 1.5 * side + 1.0
    cell = 2.0 * r + 0.05
    S = synth.box_system(n, L, H, cell, 0, density=2500e-6, kn=1e5, restitution=0.6, mu=0.4)
    vel = rng.normal(scale=60.0, size=(n, 3)).astype(np.float32)
    return [S], synth.box_walls(L, H), pos, np.full(n, r, np.float32), vel


@pytest.mark.parametrize("n", [1, 3, 33, 14208, 14209, 16384, 16385, 28417, 56833, 113664, 113665])
def test_ensemble_step_sizes(n):
    """Calls of odd and even lengths end in either buffer; a round of 16 steps
    stops early at every re-sort."""
    S, W, pos, rad, vel = ens_box(n)
    calls = (20, 9, 16, 3)
    opt = dict(law=E.LAW_LINEAR, dt=5e-6, skin=0.02)
    out, rb = [], []
    for g in (0, 1, 2):
        e = E.Ensemble(S, W, use_graph=g, **opt)
        e.set_state(pos, rad, vel)
        for c in calls:
            e.step(c)
        out.append(e.state())
        rb.append(e.num_rebuilds())
        e.close()
    if n <= 16385:
        o = EnsRestated(S, W, E.LAW_LINEAR, 5e-6, 0.02, 32, precision="f32")
        o.set_state(pos, rad, vel)
        o.step(sum(calls))
        out.append(o.state())
        rb.append(o.num_rebuilds())
    assert out[0]["status"] == 0 and len(set(rb)) == 1
    if n > 1000:
        assert rb[0] > 2
    for other in out[1:]:
        for k in ("pos", "vel", "avel"):
            np.testing.assert_array_equal(out[0][k].astype(np.float64), other[k].astype(np.float64), err_msg=k)
        np.testing.assert_array_equal(out[0]["pid"], other["pid"])


def test_mill_graph_equals_plain(tmp_path):
    """Twelve blocks: lifters turned by the last block of the step before
    (graphs) or by a kernel of their own, energy summed block by block."""
    P, st = synth.mill_project(str(tmp_path), n=3000)
    axis = float(P.wobj[0].cyl_geo.radius)
    out = []
    for g in (0, 1):
        s = device.Simulation(P, skin=0.05, use_graph=g)
        s.set_cylinder_rotation(True)
        s.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"])
        s.set_dobj_rotation(axis, axis, 50.0 * float(P.mill.RadPerStep))
        for c in (19, 40, 8):
            s.step(c)
        d = s.dobj()
        verts = [(v.x, v.y, v.z) for k in range(P.n_d) for v in d[k].vertex]
        faces = [(f.normal.x, f.normal.y, f.centroid.x, f.centroid.y, f.area)
                 for k in range(P.n_d) for f in d[k].faces]
        out.append((s.state(), s.energy(), np.array(verts), np.array(faces)))
        s.close()
    (a, ea, va, fa), (b, eb, vb, fb) = out
    for k in ("pos", "vel", "avel", "pid"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert ea[0] > 0
    np.testing.assert_array_equal(ea, eb)
    np.testing.assert_array_equal(va, vb)
    np.testing.assert_array_equal(fa, fb)
    turned = abs(67 * 50.0 * float(P.mill.RadPerStep))
    v0 = np.array([P.dobj[0].vertex[0].x - axis, P.dobj[0].vertex[0].y - axis])
    v1 = va[0, :2] - axis
    got = math.atan2(v0[0] * v1[1] - v0[1] * v1[0], v0 @ v1)
    assert abs(abs(got) - turned) < 1e-3 * turned + 1e-5


@pytest.mark.parametrize("side", [0.4, 1.1, 8.0])
def test_polyhedra_on_a_fine_mesh(side):
    """Rocks thrown on a floor of triangles: more than one window of candidate
    triangles per rock (side 0.4 cm), about one, and two in all."""
    S, _, p, r, sh, so, q = synth.mixed_box_ensemble(n_spheres=40, n_rocks=12, L=8.0, H=14.0, kn=1e5)
    L, H = 8.0, 14.0
    W = [w for k, w in enumerate(synth.box_walls(L, H)) if k != 4]
    m = int(math.ceil(L / side))
    x = np.linspace(0.0, L, m + 1)
    for i in range(m):
        for j in range(m):
            a, b = (x[i], x[j], 0.0), (x[i + 1], x[j], 0.0)
            c, d = (x[i + 1], x[j + 1], 0.0), (x[i], x[j + 1], 0.0)
            W += [E.triangle(a, b, c), E.triangle(a, c, d)]
    s = S[0]
    s.nwalls, s.tri0, s.ntris = 5, 5, len(W) - 5
    vel = np.zeros_like(p)
    vel[:, 2] = -60.0
    ens = E.Ensemble(S, W, law=E.LAW_LINEAR, dt=1e-5, skin=0.04, use_graph=1)
    o = EnsRestated(S, W, E.LAW_LINEAR, 1e-5, 0.04, 32, precision="f32")
    for e in (ens, o):
        e.set_state(p, r, vel)
        e.set_polyhedra(sh, so, q)
        e.step(1600)
    a, b = ens.state(), o.state()
    assert a["status"] == b["status"] == 0
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    np.testing.assert_array_equal(ens.orientations().astype(np.float64), o.orientations())
    rocks = so[a["pid"]] >= 0
    assert (a["vel"][rocks, 2] > 0).any()            # some have bounced
    ens.close()
    o.close()


@pytest.mark.parametrize("facets", [26, 28, 29, 70])
def test_many_planes(facets):
    """A prism of plane walls around one system (32, 33 and more walls with top,
    floor and two slanted planes: the walls are tested 32 at a time) and a plain
    box beside it, so one warp holds particles with different wall counts."""
    r, n = 0.2, 101
    pos, rng, side = lattice(n, 0.4 - 2e-4, 0.2, facets)
    c, L, H = 0.5 * side, side + 0.02, 1.5 * side + 1.0
    W, R = [], 0.5 * side + 0.01
    for k in range(facets):
        a = 2.0 * math.pi * (k + 0.5) / facets
        m = np.array([-math.cos(a), -math.sin(a), 0.0])
        W.append(E.plane(m, float(m @ [c, c, 0.0]) - R))
    W += [E.plane((0, 0, 1), 0.0), E.plane((0, 0, -1), -H)]
    for s in (1.0, -1.0):
        m = np.array([s, 0.0, 1.0]) / math.sqrt(2.0)
        W.append(E.plane(m, float(m @ [c - s * 0.5 * side, c, 0.3])))
    kw = dict(density=2500e-6, kn=1e5, restitution=0.6, mu=0.4)
    A = synth.box_system(n, L, H, 0.45, 0, **kw)
    A.nwalls = len(W)
    B = synth.box_system(n, L, H, 0.45, len(W), **kw)
    W += synth.box_walls(L, H)
    pos = np.concatenate([pos, pos])
    rad = np.full(2 * n, r, np.float32)
    vel = rng.normal(scale=60.0, size=pos.shape).astype(np.float32)
    o = EnsRestated([A, B], W, E.LAW_LINEAR, 5e-6, 0.02, 32, precision="f32")
    ens = E.Ensemble([A, B], W, law=E.LAW_LINEAR, dt=5e-6, skin=0.02, use_graph=1)
    for e in (o, ens):
        e.set_state(pos, rad, vel)
        e.step(40)
    a, b = ens.state(), o.state()
    assert a["status"] == b["status"]
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    ens.close()
    o.close()


@pytest.mark.parametrize("warps", [1, 2, 4])
def test_warps_per_polyhedron(warps):
    """A rock's tests by one warp, or by two or four in turn: rocks and balls poured on
    each other, and thrown on a floor of more than a window of triangles."""
    L, H = 8.0, 14.0
    S, W, p, r, sh, so, q = synth.mixed_box_ensemble(n_spheres=60, n_rocks=14, L=L, H=H, kn=1e5)
    x = np.linspace(0.0, L, 17)
    W = [w for k, w in enumerate(W) if k != 4]
    for i in range(16):
        for j in range(16):
            a, b = (x[i], x[j], 0.0), (x[i + 1], x[j], 0.0)
            c, d = (x[i + 1], x[j + 1], 0.0), (x[i], x[j + 1], 0.0)
            W += [E.triangle(a, b, c), E.triangle(a, c, d)]
    s = S[0]
    s.nwalls, s.tri0, s.ntris = 5, 5, len(W) - 5
    vel = np.zeros_like(p)
    vel[:, 2] = -60.0 - 6.0 * p[:, 2]                # the upper ones catch up
    ens = E.Ensemble(S, W, law=E.LAW_LINEAR, dt=1e-5, skin=0.04, use_graph=1)
    ens.set_launch(poly_warps=warps)
    o = EnsRestated(S, W, E.LAW_LINEAR, 1e-5, 0.04, 32, precision="f32")
    for e in (ens, o):
        e.set_state(p, r, vel)
        e.set_polyhedra(sh, so, q)
        e.step(1600)
    a, b = ens.state(), o.state()
    assert a["status"] == b["status"] == 0
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    np.testing.assert_array_equal(ens.orientations().astype(np.float64), o.orientations())
    ens.close()
    o.close()


@pytest.mark.parametrize("rounds", [-1, 1])
@pytest.mark.parametrize("speed", [2000.0, 600.0, 300.0, 100.0])
def test_hot_ensemble(rounds, speed):
    """Re-sorts every step, every few steps and every dozen: rounds that stop
    early, short ones, and IF nodes."""
    n, rng = 500, np.random.default_rng(5)
    g = np.arange(n)
    pos = np.stack([g % 8, g // 8 % 8, g // 64], 1) * 0.45 + 0.3
    S = synth.box_system(n, 3.9, 3.9, 0.45, 0, density=2500e-6, kn=1e6, restitution=0.9, mu=0.3)
    W = synth.box_walls(3.9, 3.9)
    vel = rng.normal(scale=speed, size=pos.shape).astype(np.float32)
    ens = E.Ensemble([S], W, law=E.LAW_LINEAR, dt=5e-6, skin=0.02, use_graph=1)
    ens.set_launch(rounds=rounds)
    o = EnsRestated([S], W, E.LAW_LINEAR, 5e-6, 0.02, 32, precision="f32")
    for e in (ens, o):
        e.set_state(pos.astype(np.float32), np.full(n, 0.2, np.float32), vel)
        for k in (33, 8, 64, 17, 20):
            e.step(k)
    a, b = ens.state(), o.state()
    assert a["status"] == b["status"]
    assert ens.num_rebuilds() == o.num_rebuilds() > 4
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    ens.close()
    o.close()


@pytest.mark.parametrize("n", [200001, 1 << 20, (1 << 20) + 1])
def test_graph_kind_by_size(n):
    """The largest box in rounds and the smallest with IF nodes; and a size
    between them (a cylinder around it: IF nodes, the box alone: rounds)."""
    S, W, pos, rad, vel = ens_box(n)
    if n == 200001:
        c = 0.5 * float(pos[:, 0].max() + 0.2)
        W = W + [E.cylinder((c, c, 0.0), (0.0, 0.0, 1.0), 3.0 * c)]
        S[0].nwalls = 7
    out = []
    for g in (0, 1):
        e = E.Ensemble(S, W, law=E.LAW_LINEAR, dt=5e-6, skin=0.02, use_graph=g)
        e.set_state(pos, rad, vel)
        for k in (9, 8):
            e.step(k)
        out.append((e.state(), e.num_rebuilds()))
        e.close()
    assert out[0][0]["status"] == out[1][0]["status"] == 0 and out[0][1] == out[1][1] > 1
    for k in ("pos", "vel", "avel", "pid"):
        np.testing.assert_array_equal(out[0][0][k], out[1][0][k], err_msg=k)


def test_launch_counts(tmp_path):
    """The launches that a step call reports, by what runs it."""
    P, st = synth.mill_project(str(tmp_path), n=3000)
    axis = float(P.wobj[0].cyl_geo.radius)
    s = device.Simulation(P, skin=0.05, use_graph=1)
    s.set_cylinder_rotation(True)
    s.set_state(st["pos"], st["vel"], st["avel"], st["type"], st["pid"])
    s.set_dobj_rotation(axis, axis, float(P.mill.RadPerStep))
    s.step(8)                       # after a new state: a gate, a move and a step each
    assert s.last_launches() == 8 * 3
    s.step(16)                      # two blocks: a gate, a move and eight steps
    assert s.last_launches() == 2 * (1 + 1 + 8)
    s.step(3)
    assert s.last_launches() == 3 * 3
    s.close()
    S, W, pos, rad, vel = ens_box(500)
    for graph, rounds, capture, steps, resort in ((0, 0, 0, 40 * 7, 5), (1, 1, 0, 2 + 6 + 40, 7),
                                                  (1, -1, 0, 5 * 9, 5), (2, 0, 0, 3, 7),
                                                  (2, 0, 1, 2 + 6 + 40, 7), (2, -1, 1, 5 * 9, 5)):
        e = E.Ensemble(S, W, law=E.LAW_LINEAR, dt=5e-6, skin=0.02, use_graph=graph,
                       capture_forces=capture)
        e.set_launch(rounds=rounds)
        e.set_state(pos, rad)
        e.step(40)
        assert (e.last_launches(), e.rebuild_kernels()) == (steps, resort), (graph, rounds, capture)
        e.close()


# (size of the triangle, radius, centre): spheres that touch a vertex of a small
# triangle at the origin by a few 1e-8 cm, where FP32 rounds the distance to the
# triangle's bounding sphere beyond the sum of the radii
GRAZING = [
    (0.0012349095360439084, 1.4137132167816162, (1.4149479866027832, -0.00039765366818755865, 0.00037886638892814517)),
    (0.0013415310415354174, 1.9994114637374878, (2.0007522106170654, 0.0010979132493957877, 0.0013439931208267808)),
    (0.0025264999515147773, 1.4134680032730103, (1.4159938097000122, 0.0010431538103148341, 0.000926253735087812)),
    (0.0002965804566498865, 1.999942421913147, (2.0002386569976807, 0.0009980620816349983, -0.0005503043648786843)),
    (0.0007389509463619639, 1.999290943145752, (2.0000290870666504, -0.0016199497040361166, 0.0005662687472067773)),
    (6.981820006969034e-05, 0.49996626377105713, (0.5000360608100891, -0.0001299064460908994, -1.1633491340035107e-05)),
    (5.280388288221428e-05, 0.9999672770500183, (1.0000196695327759, 0.000817042775452137, 0.00034754013177007437)),
    (6.595577163958962e-05, 0.9999799728393555, (1.0000455379486084, -0.0008272947743535042, 0.0002528926415834576)),
]


def test_grazing_contact_with_a_small_triangle():
    S, W, pos, rad = [], [], [], []
    for k, (s, r, p) in enumerate(GRAZING):
        W.append(E.triangle((s, 0, 0), (-0.5 * s, 0.8 * s, 0), (-0.5 * s, -0.8 * s, 0)))
        y = synth.box_system(1, 8.0, 8.0, 4.1, 0, density=2500e-6, kn=1e8, restitution=0.6,
                             mu=0.4, gravity=(0.0, 0.0, 0.0))
        y.nwalls, y.tri0, y.ntris = 0, k, 1
        for a in range(3):
            y.origin[a] = -4.1
        S.append(y)
        pos.append(p)
        rad.append(r)
    pos, rad = np.array(pos, np.float32), np.array(rad, np.float32)
    ens = E.Ensemble(S, W, law=E.LAW_LINEAR, dt=1e-4, skin=0.01, use_graph=0)
    o = EnsRestated(S, W, E.LAW_LINEAR, 1e-4, 0.01, 32, precision="f32")
    for e in (ens, o):
        e.set_state(pos, rad)
        e.step(1)
    a, b = ens.state(), o.state()
    assert a["status"] == b["status"] == 0
    assert (b["vel"][:, 0] > 0).all()
    np.testing.assert_array_equal(a["vel"].astype(np.float64), b["vel"])
    ens.close()
    o.close()


@pytest.mark.parametrize("grid", [0, 1])
def test_new_volume_objects_keep_the_world_objects(tmp_path, grid):
    """blaze_update_dobj replaces the volume objects and nothing else: without
    the per-cell wall lists (also with polyhedra, or moving walls) the particles
    lost every world object."""
    r, n = 0.1, 257
    P, _ = synth.box_project(str(tmp_path), n_side=(2, 2, 2), radius=r)
    P.sim_info.Num_Particles = n
    pos, rng, _ = lattice(n, 0.1995, 0.0995, n)       # touching the walls and each other
    vel = rng.normal(scale=10.0, size=(n, 3)).astype(np.float32)
    avel, ty, pid = np.zeros_like(vel), np.zeros(n, np.uint32), np.arange(n, dtype=np.int32)
    sim = device.Simulation(P, wall_grid=grid)
    ref = Restated("f32").init(P.sim_info, P.wobj, P.n_w, P.pobj, P.n_p, P.dobj, P.n_d)
    for s in (sim, ref):
        s.set_state(pos, vel, avel, ty, pid)
    sim.update_dobj(P.dobj, P.n_d)
    sim.step(5)
    ref.step(5)
    a, b = sim.state(), ref.state()
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    sim.close()
