"""The sphere list build (pairs met once, records ranked by key, partner lists by
rank) against the oracle's lists: particles of uneven size with long lists (more
candidates than a record holds), few cells along an axis, periodic faces on every
axis, cells larger than needed, and ids in an order unlike the positions'."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

FLAGS = dict(fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1)


def _cloud(n, box, periodic, seed, big=0, cell=0.0, skin=0.05):
    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1, **FLAGS)
    w.params.bounds_hi[:] = [box] * 3
    for q, wall in enumerate(w.surfaces):
        wall["offset"] = box if q % 2 else 0.0
    rng = np.random.default_rng(seed)
    arr = W.empty_particles(n)
    for f in ("rx", "ry", "rz"):
        arr[f] = rng.uniform(0.0, box, n)
    r = rng.uniform(0.25, 0.4, n)
    r[:big] = 2.0
    arr["radius"], arr["mass"] = r, 2.0 * r ** 3
    for f in ("inertiax", "inertiay", "inertiaz"):
        arr[f] = 0.4 * arr["mass"] * r * r
    arr["qw"], arr["homothety"] = np.ones(n), np.ones(n)
    for f in ("vx", "vy", "vz"):
        arr[f] = rng.uniform(-0.5, 0.5, n)
    arr["id"] = rng.permutation(np.arange(n, dtype=np.uint64) * np.uint64(7) + np.uint64(3))
    w.particles = arr
    w.params.periodic[:] = periodic
    w.params.cell_size = cell
    w.params.rcut_inc = skin
    w.params.config.kn = w.params.config_driver.kn = 10.0
    if any(periodic):
        w.surfaces = []
    return w


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("n,box,periodic,big,cell,skin", [
    (1, 4.0, (0, 0, 0), 0, 0.0, 0.05), (2, 3.0, (1, 1, 1), 0, 0.0, 0.05), (33, 2.6, (1, 1, 1), 0, 0.0, 0.05),
    (700, 6.0, (1, 0, 1), 0, 0.0, 0.3), (900, 13.0, (0, 1, 0), 3, 0.0, 0.05), (1500, 9.0, (0, 0, 0), 0, 4.0, 0.05),
    (257, 1.5, (0, 0, 0), 0, 0.0, 0.2)])
def test_lists_match_oracle(native_lib, n, box, periodic, big, cell, skin, graph):
    w = _cloud(n, box, periodic, 80 + n, big, cell, skin)
    w.params.graph_step = graph
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    assert_same_list(g.interactions(), o.interactions())
    for s in (g, o):
        s.step(60)
    assert g.rebuild_count() == o.rebuild_count()
    assert_same_list(g.interactions(), o.interactions())
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
