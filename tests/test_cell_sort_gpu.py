"""The re-sort by cell and the neighbour search on it, against the definition:
a stable sort by the reference's hash (particles outside the grid, then parked
ones, behind the others in their order) and the clamped 27 cells scanned in
y, z, x order, at the sizes where the counting sort and the row search can go
wrong: one block of particles and its edges, a tile of cells and its edges, more
tiles than the scan has blocks, radii that reach a few or all of their cells,
grids whose hash aliases (x + z ncz + y ncx ncz with ncx != ncz), grids too
small to leave cells out of the search, crowded cells."""
import numpy as np
import pytest

from blaze import device, synth
from blaze import types as T

pytestmark = pytest.mark.gpu

F = np.float32


def definition(pos, pid, rad, origin, cell, nc, skin):
    """(sorted order of the input, list per sorted particle)"""
    n = len(pos)
    g = np.floor((pos - origin) / cell).astype(np.int64)
    inside = np.all((g >= 0) & (g < nc), axis=1)
    big = 1 << 40
    key = g[:, 0] + g[:, 2] * nc[2] + g[:, 1] * nc[0] * nc[2]
    key = np.where(pid < 0, big + 1, np.where(inside, key, big))
    order = np.argsort(key, kind="stable")
    p, k, gs, live = pos[order], key[order], g[order], (pid >= 0)[order]
    bucket = {}
    for i in range(n):
        if k[i] < big:
            bucket.setdefault(int(k[i]), []).append(i)
    lists = []
    rs = np.broadcast_to(np.asarray(rad, F), n)[order]
    for i in range(n):
        out = []
        if k[i] < big and live[i]:
            for y in range(max(0, gs[i, 1] - 1), min(nc[1], gs[i, 1] + 2)):
                for z in range(max(0, gs[i, 2] - 1), min(nc[2], gs[i, 2] + 2)):
                    for x in range(max(0, gs[i, 0] - 1), min(nc[0], gs[i, 0] + 2)):
                        for j in bucket.get(int(x + z * nc[2] + y * nc[0] * nc[2]), ()):
                            if j == i:
                                continue
                            d = p[i] - p[j]
                            sr = rs[i] + rs[j]
                            d2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
                            if skin > 0:
                                reach = sr + F(skin)
                                hit = d2 < (reach * reach) * (F(1) + F(2.0 ** -20))
                            else:
                                hit = np.sqrt(d2) - sr < 0
                            if hit:
                                out.append(j)
        lists.append(out)
    return order, lists


@pytest.mark.parametrize("n,nc,fill,skin", [
    (1, (3, 3, 3), 1.0, 0.0), (255, (7, 7, 7), 0.5, 0.0), (256, (16, 16, 16), 0.3, 0.0),
    (257, (15, 13, 21), 0.3, 0.0), (3000, (17, 15, 16), 0.9, 0.0), (3000, (16, 17, 16), 1.2, 0.05),
    (700, (12, 5, 2), 0.9, 0.0), (700, (2, 9, 11), 0.9, 0.0), (400, (1, 1, 1), 0.1, 0.0),
    (2000, (64, 2, 64), 1.1, 0.0), (1500, (9, 9, 9), 1.3, 0.1), (5000, (40, 40, 40), 1.0, 0.0),
    (2000, (211, 204, 210), 1.0, 0.0), (3000, (211, 204, 210), 0.06, 0.0)])
def test_order_and_list_by_definition(tmp_path, n, nc, fill, skin):
    rad = 0.1
    P, _ = synth.box_project(str(tmp_path), n_side=(2, 2, 2), radius=rad)
    cell = np.full(3, F(2 * rad + skin), F)
    if nc == (1, 1, 1):
        cell = np.full(3, F(3.0), F)
    check(P, n, nc, fill, skin, cell, np.array([rad]))


@pytest.mark.parametrize("n,nc,fill,skin", [
    (3000, (17, 15, 16), 0.6, 0.0), (2000, (8, 9, 6), 0.9, 0.0), (1000, (6, 5, 7), 0.9, 0.0),
    (1000, (5, 7, 9), 0.9, 0.0), (2500, (12, 6, 12), 0.9, 0.1)])
def test_mixed_radii(tmp_path, n, nc, fill, skin):
    """Small spheres reach few of their 27 cells: those are left out only where
    the grid has six cells along x and z, and never with a partner in reach."""
    radii = np.array([0.03, 0.06, 0.1], F)
    S = synth.box_system(8, 1.0, 1.0, 0.25, 0, density=2500e-6, kn=1e5)
    P, _ = synth.box_system_project(str(tmp_path), "Box", S, 1.0, 1.0, radii, 2500.0)
    got = np.array([P.pobj[k].radius for k in range(P.n_p)], F)
    np.testing.assert_allclose(got, radii, rtol=1e-6)
    check(P, n, nc, fill, skin, np.full(3, F(0.2) + F(skin), F), got)


def check(P, n, nc, fill, skin, cell, radii):
    rng = np.random.default_rng(n + nc[0])
    origin = np.array([-0.3, 0.2, 5.0], F)
    nc = np.array(nc)
    # a cloud over part of the grid, some of it outside, some of it parked
    pos = (origin + rng.uniform(-0.05, 1.0, (n, 3)) * nc * cell * min(1.05, fill)).astype(F)
    pid = np.where(rng.random(n) < 0.1, -1, np.arange(n)).astype(np.int32)
    if n == 1:
        pos[0], pid[0] = origin + 0.5 * cell, 0
    kind = rng.integers(0, len(radii), n).astype(np.uint32)
    si = P.sim_info
    si.Num_Particles = n
    for name, v in (("worldOrigin", origin), ("cellSize", cell)):
        for a, x in zip("xyz", v):
            setattr(getattr(si, name), a, float(x))
    for a, x in zip("xyz", nc):
        setattr(si.num_NNCells, a, int(x))
        setattr(si.Force_Field, a, 0.0)
    sim = device.Simulation(sim_info=si, wobj=None, n_w=0, pobj=P.pobj, n_p=P.n_p, skin=skin)
    sim.set_state(pos, ptype=kind, pid=pid)
    sim.step(1)
    status = sim.sync()
    nn, lst = sim.nlist()
    got = sim.state()["pid"]
    sim.close()
    order, lists = definition(pos, pid, radii[kind], origin, cell, nc, skin)
    np.testing.assert_array_equal(got, pid[order])
    full = any(len(x) > 32 for x in lists)
    assert bool(status & 1) == full
    for i, x in enumerate(lists):
        assert nn[i] == min(len(x), 32)
        np.testing.assert_array_equal(lst[i, :nn[i]], x[:32])
