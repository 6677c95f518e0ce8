"""Mesh candidates of spheres on the GPU against the oracle's lists: the bins' items
of 32 spheres dealt to the threads of a block, two mesh drivers, a vertex where
48 triangles meet (spheres with more candidates than a record holds), numbers of
spheres that leave threads and blocks partly empty, the mesh far from the origin, both
list builds of the FP32 broad phase and the FP64 one."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from exadem_gb300.stl import build_shape
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu


def _fan(k, radius):
    t = np.linspace(0.0, 2.0 * np.pi, k, endpoint=False)
    rim = [(radius * np.cos(x), radius * np.sin(x), 0.0) for x in t]
    return [((0.0, 0.0, 0.4), rim[q], rim[(q + 1) % k]) for q in range(k)]


def _fan_mesh(k, radius, center):
    shp = build_shape([np.asarray(t) for t in _fan(k, radius)])
    return dict(vertices=shp["vertices"], edges=shp["edges"], faces=shp["faces"], minkowski=0.05, center=center,
                quat=(1.0, 0.0, 0.0, 0.0))


def _cloud(n, origin, **flags):
    w = W.spheres_mesh_terrain(n=8, seed=5, fused_step=1, fp32_contact_screen=1, **flags)
    lo = np.asarray((origin, -origin, origin))
    w.params.bounds_lo[:] = lo
    w.params.bounds_hi[:] = lo + 16.0
    w.surfaces = []
    w.meshes = [_fan_mesh(48, 6.0, tuple(lo + (8.0, 8.0, 3.0))), _fan_mesh(5, 7.0, tuple(lo + (8.0, 8.0, 6.0)))]
    rng = np.random.default_rng(n)
    arr = W.empty_particles(n)
    for d, f in enumerate(("rx", "ry", "rz")):
        arr[f] = lo[d] + rng.uniform((1.0, 1.0, 2.0)[d], (15.0, 15.0, 8.0)[d], n)
    near = slice(0, max(1, n // 8))  # about the vertex where the triangles meet
    for d, f in enumerate(("rx", "ry", "rz")):
        arr[f][near] = lo[d] + rng.uniform((7.6, 7.6, 3.5)[d], (8.4, 8.4, 4.2)[d], len(arr[f][near]))
    r = rng.uniform(0.15, 0.3, n)
    arr["radius"], arr["mass"] = r, 2.0 * r ** 3
    for f in ("inertiax", "inertiay", "inertiaz"):
        arr[f] = 0.4 * arr["mass"] * r * r
    arr["qw"], arr["homothety"] = np.ones(n), np.ones(n)
    for f in ("vx", "vy", "vz"):
        arr[f] = rng.uniform(-0.5, 0.5, n)
    arr["id"] = rng.permutation(np.arange(n, dtype=np.uint64))
    w.particles = arr
    w.params.config.kn = w.params.config_driver.kn = 10.0
    return w


@pytest.mark.parametrize("n,origin,fp32,graph,cells", [
    (1, 0.0, 1, 1, 0), (7, 0.0, 1, 1, 0), (9, 0.0, 1, 0, 0), (33, 0.0, 1, 1, 0), (600, 0.0, 1, 1, 0),
    (600, 4096.0, 1, 1, 0), (601, 0.0, 1, 0, 1), (600, 0.0, 0, 0, 0)])
def test_mesh_candidates_match_oracle(native_lib, n, origin, fp32, graph, cells):
    w = _cloud(n, origin, fp32_broad_phase=fp32, graph_step=graph)
    g, o = pair(w)
    if cells:
        g.set_sphere_cell_broad_phase(1)
    for s in (g, o):
        s.first_iteration()
    lst = g.interactions()
    assert_same_list(lst, o.interactions())
    if n >= 600:
        mesh = np.isin(lst["type"], (7, 8, 9))
        assert np.unique(lst["owner_id"][mesh], return_counts=True)[1].max() > 16
    for s in (g, o):
        s.step(60)
    assert g.rebuild_count() == o.rebuild_count()
    assert_same_list(g.interactions(), o.interactions())
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
