"""Rotations that a block puts off to its end (more particles than a warp a scheduler,
few of a warp's lanes rotating) against the oracle, bit for bit: no, few, half and all
particles spinning, at random and in runs of whole warps; spheres in the host-launched
and the graph step, polyhedra with rebuilds raised by a spinning particle's vertices."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

N = 20011  # above 128 particles an SM


def _spin(a, share, runs, seed, rate):
    rng = np.random.default_rng(seed)
    n = len(a["rx"])
    on = rng.random(n) < share
    if runs:
        on = np.repeat(rng.random((n + 63) // 64) < share, 64)[:n]
    for f in ("vrotx", "vroty", "vrotz"):
        a[f] = np.where(on, rng.uniform(-rate, rate, n), 0.0)


@pytest.mark.parametrize("share,runs,graph", [(0.0, 0, 1), (0.05, 0, 1), (0.05, 0, 0), (0.5, 0, 1), (0.5, 1, 1),
                                              (1.0, 0, 1)])
def test_spheres(native_lib, share, runs, graph):
    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1, fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1,
                      graph_step=graph)
    side = 28
    box = side * 1.3
    w.params.bounds_hi[:] = [box] * 3
    for q, wall in enumerate(w.surfaces):
        wall["offset"] = box if q % 2 else 0.0
    rng = np.random.default_rng(7)
    a = W.empty_particles(N)
    cell = rng.permutation(side ** 3)[:N]
    for d, f in enumerate(("rx", "ry", "rz")):
        a[f] = (cell // side ** d % side + 0.5) * 1.3 + rng.uniform(-0.2, 0.2, N)
    r = rng.uniform(0.4, 0.55, N)
    a["radius"], a["mass"] = r, 2.0 * r ** 3
    for f in ("inertiax", "inertiay", "inertiaz"):
        a[f] = 0.4 * a["mass"] * r * r
    a["qw"], a["homothety"] = np.ones(N), np.ones(N)
    a["id"] = np.arange(N, dtype=np.uint64)
    _spin(a, share, runs, 8, 5.0)
    w.particles = a
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(1)
        s.step(12)
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))


@pytest.mark.parametrize("share,runs", [(0.0, 0), (0.05, 0), (0.5, 1), (1.0, 0)])
def test_polyhedra(native_lib, share, runs):
    w = W.polyhedra_lattice(nx=28, ny=28, nz=26, spacing=2.6, seed=3, fused_step=1, fp32_broad_phase=1,
                            fp32_contact_screen=1, dt=1e-3, skin=0.05)
    _spin(w.particles, share, runs, 9, 4.0)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(1)
        s.step(12)
    assert g.rebuild_count() == o.rebuild_count()
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
