"""Walls far from the corner of a wide domain: the lists against the oracle's for a
plane through the origin (straight and oblique) and a cylinder about an axis through
it, where the coordinates are small against the domain's lower bounds, and particles
that sit 1e-9 to 1e-2 of the skin inside and outside the reach."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair

pytestmark = pytest.mark.gpu

SKIN = 0.05


def _gap(rng, n, r):
    return r + SKIN + rng.choice((-1.0, 1.0), n) * SKIN * 10.0 ** rng.uniform(-9.0, -2.0, n)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("wall", ["plane", "oblique", "cylinder"])
@pytest.mark.parametrize("lo", [(-100.0, -100.0, -6.0), (-1000.0, -7.0, -1000.0), (-4000.0, -6.5, -5.3),
                                (4000.0, 40.0, 700.0)])
def test_spheres(native_lib, lo, wall, graph):
    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1, fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1,
                      graph_step=graph)
    n = 400
    rng = np.random.default_rng(n + int(abs(lo[0])) + len(wall))
    r = rng.uniform(0.3, 0.6, n)
    at = np.maximum(0.0, np.asarray(lo)) + np.where(np.asarray(lo) > 0.0, 8.0, 0.0)  # the wall's point
    w.params.bounds_lo[:] = lo
    w.params.bounds_hi[:] = at + 8.0
    p = rng.uniform(-2.2, 2.2, (n, 3))
    side = rng.choice((-1.0, 1.0), n)
    w.surfaces, w.cylinders = [], []
    if wall == "cylinder":  # about the y axis
        t = rng.uniform(0.0, 2.0 * np.pi, n)
        d = 4.5 - _gap(rng, n, r)
        p[:, 0], p[:, 2] = d * np.cos(t), d * np.sin(t)
        w.cylinders = [dict(radius=4.5, axis=(1.0, 0.0, 1.0), center=tuple(at))]
    else:
        nrm = np.asarray((1.0, 0.0, 0.0) if wall == "plane" else (0.6, 0.64, -0.48))
        p += (side * _gap(rng, n, r) - p @ nrm)[:, None] * nrm
        w.surfaces = [dict(offset=float(at @ nrm), normal=tuple(nrm))]
    p += at
    arr = W.empty_particles(n)
    for k, f in enumerate(("rx", "ry", "rz")):
        arr[f] = np.ascontiguousarray(p[:, k])
    arr["radius"], arr["mass"] = r, 2.0 * r ** 3
    for f in ("inertiax", "inertiay", "inertiaz"):
        arr[f] = 0.4 * arr["mass"] * r * r
    arr["qw"], arr["homothety"] = np.ones(n), np.ones(n)
    arr["id"] = np.arange(n, dtype=np.uint64)
    w.particles = arr
    w.params.rcut_inc = SKIN
    w.params.config.kn = w.params.config_driver.kn = 1.0
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    lst = o.interactions()
    walls = np.isin(lst["type"], (4, 5)).sum()
    assert n // 4 < walls < 3 * n // 4  # about half of them inside the reach
    assert_same_list(g.interactions(), lst)
    for s in (g, o):  # the rebuild inside a step
        s.update_particle_neighbors()
        s.step(2)
    assert_same_list(g.interactions(), o.interactions())


@pytest.mark.parametrize("wall", ["plane", "cylinder"])
@pytest.mark.parametrize("lo", [(-1000.0, -1000.0, -8.0), (-4000.0, -8.5, -9.3)])
def test_polyhedra(native_lib, lo, wall):
    """A cube's corner turned to the wall, so the wall is at the end of the cube's reach."""
    w = W.polyhedra_lattice(nx=8, ny=8, nz=1, spacing=4.0, seed=3, fused_step=1, fp32_broad_phase=1,
                            fp32_contact_screen=1)
    a = w.particles
    n = len(a["rx"])
    rng = np.random.default_rng(int(-lo[0]))
    a["type"][:] = 0
    a["homothety"] = np.ones(n)
    corner = np.sqrt(0.75)
    shape = w.shapes[0]
    assert np.allclose(np.abs(np.asarray(shape["vertices"])), 0.5)
    w.params.bounds_lo[:] = lo
    w.params.bounds_hi[:] = (8.0, 8.0, 8.0)
    gap = corner + _gap(rng, n, float(shape["radius"]))
    p = np.stack([a["rx"], a["ry"], a["rz"]], 1)
    if wall == "plane":  # x = 0
        out = np.tile((-1.0, 0.0, 0.0), (n, 1))
        p[:, 0] = gap
        p[:, 1:] = np.stack([np.arange(n) % 8, np.arange(n) // 8], 1) * 0.8 - 2.8
        w.surfaces, w.cylinders = [dict(offset=0.0, normal=(1.0, 0.0, 0.0))], []
    else:  # about the z axis
        t = np.arange(n) * (2.0 * np.pi / 8)
        d = 3.5 - gap
        p[:, 0], p[:, 1], p[:, 2] = d * np.cos(t), d * np.sin(t), (np.arange(n) // 8) * 0.8 - 2.8
        out = np.stack([np.cos(t), np.sin(t), np.zeros(n)], 1)
        w.surfaces, w.cylinders = [], [dict(radius=3.5, axis=(1.0, 1.0, 0.0), center=(0.0, 0.0, 0.0))]
    c = np.full(3, 1.0 / np.sqrt(3.0))  # q turns the corner (1, 1, 1) to out
    q = np.concatenate([1.0 + out @ c[:, None], np.cross(np.tile(c, (n, 1)), out)], 1)
    q /= np.linalg.norm(q, axis=1)[:, None]
    for k, f in enumerate(("qw", "qx", "qy", "qz")):
        a[f] = np.ascontiguousarray(q[:, k])
    for k, f in enumerate(("rx", "ry", "rz")):
        a[f] = np.ascontiguousarray(p[:, k])
    w.params.rcut_inc = SKIN
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    lst = o.interactions()
    walls = np.isin(lst["type"], (4, 5)).sum()
    assert n // 4 < walls < 3 * n // 4
    assert_same_list(g.interactions(), lst)
