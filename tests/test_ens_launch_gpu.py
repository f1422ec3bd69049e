"""The ensemble step's builds and launch shapes, forced at small sizes
(blaze_ens_set_launch), against the restatement: full warps whose contacts take
several passes of the shared buffer, wall contacts that fill it, the builds at
64 and 80 registers, and the step graphs with a conditional node before every
step, for planes, meshes, turning drums, mixed charges and recorded runs."""
import math

import numpy as np
import pytest

from bindings import EnsRestated
from blaze import ensemble as E
from blaze import synth
from test_ensemble_gpu import DT, SKIN, mesh_silo, turning_drum
from test_mixed_gpu import CASES as MIXED

pytestmark = pytest.mark.gpu

LAUNCH = [dict(warp_particles=32, registers=64), dict(warp_particles=32, registers=80),
          dict(warp_particles=8, registers=64), dict(rounds=-1, warp_particles=16)]


def bed(n, gap=2e-4, roll=0.01):
    """n sites of a face-centred lattice, neighbours overlapping by `gap`, in a box."""
    r = 0.2
    s = (2.0 * r - gap) / math.sqrt(2.0)
    m = int(math.ceil((2.0 * n) ** (1.0 / 3.0)))
    g = np.arange(m * m * 4 * m)
    x, y, z = g % m, g // m % m, g // (m * m)
    k = np.flatnonzero((x + y + z) % 2 == 0)[:n]
    pos = np.stack([x[k], y[k], z[k]], 1) * s + r - 1e-4
    L, H = (m - 1) * s + 2.0 * r, float(pos[:, 2].max()) + 1.0
    rng = np.random.default_rng(n)
    pos = (pos + rng.uniform(-2e-5, 2e-5, pos.shape))[rng.permutation(n)].astype(np.float32)
    S = synth.box_system(n, L, H, 2.0 * r + 0.05, 0, density=2500e-6, kn=1e5, youngs=1e5,
                         restitution=0.6, mu=0.4, mu_roll=roll)
    vel = rng.normal(scale=20.0, size=pos.shape).astype(np.float32)
    return S, synth.box_walls(L, H), pos, np.full(n, r, np.float32), vel


def most_contacts(pos, rad, pid):
    """The most contacts of 32 particles that follow each other in memory."""
    d = pos[:, None, :].astype(np.float64) - pos[None]
    c = ((d * d).sum(2) < (rad[:, None] + rad[None]) ** 2).sum(1) - 1
    c = c[pid]
    return max(int(c[k:k + 32].sum()) for k in range(0, len(c), 32))


def equal(a, b):
    assert a["status"] == b["status"] == 0
    for k in ("pos", "vel", "avel"):
        np.testing.assert_array_equal(a[k].astype(np.float64), b[k], err_msg=k)
    np.testing.assert_array_equal(a["pid"], b["pid"])


def both(S, W, pos, rad, vel, law, launch, steps, dt=DT, skin=SKIN, poly=None):
    ens = E.Ensemble(S, W, law=law, dt=dt, skin=skin, use_graph=1)
    ens.set_launch(**launch)
    o = EnsRestated(S, W, law, dt, skin, 32, precision="f32")
    for e in (ens, o):
        e.set_state(pos, rad, vel)
        if poly:
            e.set_polyhedra(*poly)
        for k in steps:
            e.step(k)
    a, b = ens.state(), o.state()
    equal(a, b)
    assert ens.num_rebuilds() == o.num_rebuilds()
    if poly:
        np.testing.assert_array_equal(ens.orientations().astype(np.float64), o.orientations())
    ens.close()
    o.close()
    return a


@pytest.mark.parametrize("launch", LAUNCH)
@pytest.mark.parametrize("law", [E.LAW_LINEAR, E.LAW_HERTZ_MINDLIN])
def test_contacts_beyond_one_pass(law, launch):
    S, W, pos, rad, vel = bed(500)
    a = both([S], W, pos, rad, vel, law, launch, (1, 39), dt=5e-6, skin=0.02)
    # three passes of 96 contacts with full warps, the last not full
    assert most_contacts(pos, rad, a["pid"]) > 200


@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("law", [E.LAW_LINEAR, E.LAW_HERTZ_MINDLIN])
def test_wall_contacts_beyond_the_buffer(law, mesh):
    """A layer of 64 spheres on a floor that is there four times: 128 wall
    contacts in a warp, whose buffer holds 64."""
    r = 0.2
    g = np.arange(64)
    pos = np.stack([(g % 8) * 0.41 + 0.3, (g // 8) * 0.41 + 0.3, np.full(64, r - 1e-4)], 1)
    rng = np.random.default_rng(3)
    pos[:, 2] -= rng.uniform(0.0, 5e-5, 64)
    S = synth.box_system(64, 3.6, 3.0, 0.45, 0, density=2500e-6, kn=1e5, youngs=1e5,
                         restitution=0.6, mu=0.4, mu_roll=0.01)
    W = synth.box_walls(3.6, 3.0)
    if mesh:
        W = [w for k, w in enumerate(W) if k != 4]
        S.nwalls = 5
        W += [E.triangle((-9.0, -9.0, 0.0), (20.0, -9.0, 0.0), (-9.0, 20.0, 0.0))] * 4
        S.tri0, S.ntris = 5, 4
    else:
        W += [E.plane((0, 0, 1), 0.0)] * 3
        S.nwalls = 9
    vel = rng.normal(scale=20.0, size=pos.shape).astype(np.float32)
    for launch in (dict(warp_particles=32, registers=64), dict(warp_particles=32, registers=80)):
        both([S], W, pos.astype(np.float32), np.full(64, r, np.float32), vel, law, launch, (1, 19),
             dt=5e-6, skin=0.02)


@pytest.mark.parametrize("launch", LAUNCH)
@pytest.mark.parametrize("law", [E.LAW_LINEAR, E.LAW_HERTZ_MINDLIN])
@pytest.mark.parametrize("case", [mesh_silo, turning_drum])
def test_meshes(case, law, launch):
    S, W, p, r, v = case()
    both(S, W, p, r, v, law, launch, (1, 9, 190))


@pytest.mark.parametrize("launch", LAUNCH)
@pytest.mark.parametrize("name", sorted(MIXED))
def test_mixed_charges(name, launch):
    S, W, p, r, sh, so, q = MIXED[name]()
    v = np.zeros_like(p)
    v[:, 1 if name == "drum" else 2] = -60.0
    both(S, W, p, r, v, E.LAW_LINEAR, launch, (1, 9, 390), dt=1e-5, skin=0.04, poly=(sh, so, q))


@pytest.mark.parametrize("wp", [4, 32])
def test_recorded_run(wp):
    """Reverse mode through a dense bed: the recording step's histories of a
    full warp.  The bound is the reverse sweep's against the FP32 restatement
    (the order of its sums differs), as in test_adjoint_gpu.py."""
    S, W, pos, rad, vel = bed(200, roll=0.0)
    steps = 30
    rng = np.random.default_rng(1)
    wx, wv = rng.normal(size=pos.shape), 1e-2 * rng.normal(size=pos.shape)
    ens = E.Ensemble([S], W, law=E.LAW_LINEAR, dt=5e-6, skin=0.02, use_graph=0)
    ens.set_launch(warp_particles=wp)
    ens.set_state(pos, rad, vel)
    adj = E.Adjoint(ens, steps, 16)
    assert adj.forward() == 0
    a = ens.state()
    got = adj.backward(wx[a["pid"]], wv[a["pid"]], None)
    o = EnsRestated([S], W, E.LAW_LINEAR, 5e-6, 0.02, 32, precision="f32")
    o.set_state(pos, rad, vel)
    assert o.adj_record(steps) == 0
    b = o.state()
    np.testing.assert_array_equal(a["pos"].astype(np.float64), b["pos"])
    assert most_contacts(pos, rad, a["pid"]) > 200
    want = o.adj_reverse(wx[b["pid"]], wv[b["pid"]], np.zeros(pos.shape))
    for g, w in zip(got, want):
        w = np.asarray(w)
        np.testing.assert_allclose(np.asarray(g).reshape(w.shape), w, rtol=0,
                                   atol=1e-4 * np.abs(w).max())
    adj.close()
    ens.close()
    o.close()


@pytest.mark.parametrize("side", [0.09, 0.15, 0.3, 0.8])
def test_warps_that_lie_on_a_mesh(side):
    """A layer on a floor of triangles: lists of several windows, tested by the
    warp or by each lane (shorter ones), also past their first 32 entries, and
    contacts on faces, edges and vertices."""
    r, n = 0.2, 64
    g = np.arange(n)
    rng = np.random.default_rng(7)
    pos = np.stack([(g % 8) * 0.41 + 0.3, (g // 8) * 0.41 + 0.3, np.full(n, r - 2e-4)], 1)
    pos[:, :2] += rng.uniform(-2e-3, 2e-3, (n, 2))
    m = int(math.ceil(3.6 / side))
    x = np.linspace(0.0, 3.6, m + 1)
    z = 0.02 * ((np.add.outer(np.arange(m + 1), np.arange(m + 1)) % 3) == 0) if side > 0.2 else \
        np.zeros((m + 1, m + 1))
    W = [w for k, w in enumerate(synth.box_walls(3.6, 3.0)) if k != 4]
    for i in range(m):
        for j in range(m):
            a, b = (x[i], x[j], z[i, j]), (x[i + 1], x[j], z[i + 1, j])
            c, d = (x[i + 1], x[j + 1], z[i + 1, j + 1]), (x[i], x[j + 1], z[i, j + 1])
            W += [E.triangle(a, b, c), E.triangle(a, c, d)]
    S = synth.box_system(n, 3.6, 3.0, 0.45, 0, density=2500e-6, kn=1e5, restitution=0.6, mu=0.4)
    S.nwalls, S.tri0, S.ntris = 5, 5, len(W) - 5
    vel = rng.normal(scale=20.0, size=pos.shape).astype(np.float32)
    for wp in (4, 32):
        both([S], W, pos.astype(np.float32), np.full(n, r, np.float32), vel, E.LAW_LINEAR,
             dict(warp_particles=wp), (1, 60), dt=5e-6, skin=0.02)
