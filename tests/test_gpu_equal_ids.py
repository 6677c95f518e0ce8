"""Particles that share an id (nothing checks that ids differ, and the list's order and
its history go by them): the FP32 list builds, which rank an owner's entries, against
the FP64 ones, which sort them as they are met.  The lists, the histories and every
bit of the particles in their slots are the same: spheres in walls and across periodic
faces, more entries than a record holds, mesh candidates, and polyhedra."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.test_gpu_mesh_lists import _cloud as mesh_cloud
from tests.test_gpu_sphere_lists import _cloud as sphere_cloud

pytestmark = pytest.mark.gpu


def _share(w, k, seed):
    n = w.n
    w.particles["id"] = np.random.default_rng(seed).permutation(np.arange(n, dtype=np.uint64) // np.uint64(k))


def _both(w, steps):
    runs = []
    for fp32 in (1, 0):
        w.params.fp32_broad_phase = fp32
        s = w.build()
        s.first_iteration()
        lists = [s.interactions()]
        s.step(steps)
        lists.append(s.interactions())
        runs.append((lists, s.particles(sort_by_id=False), s.rebuild_count(), s.simulation_state()))
        s.close()
    (la, pa, ra, sa), (lb, pb, rb, sb) = runs
    assert ra == rb and sa["n_active_interactions"] == sb["n_active_interactions"] > 0
    for a, b in zip(la, lb):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    for k in pa:
        assert np.array_equal(np.asarray(pa[k]).view(np.uint8), np.asarray(pb[k]).view(np.uint8)), k
    return la[0]


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("k", [2, 5, 400])
@pytest.mark.parametrize("n,box,periodic,skin", [
    (60, 2.7, (1, 1, 1), 0.05), (700, 6.0, (1, 0, 1), 0.3), (800, 8.0, (0, 0, 0), 0.05), (200, 1.6, (0, 0, 0), 0.2)])
def test_spheres(native_lib, n, box, periodic, skin, k, graph):
    w = sphere_cloud(n, box, periodic, 30 + n, 0, 0.0, skin)
    w.params.graph_step = graph
    _share(w, min(k, n), n + k)
    lst = _both(w, 40)
    key = np.stack([lst["owner_id"], lst["partner_id"], lst["type"]])
    assert len(np.unique(key, axis=1).T) < key.shape[1]


@pytest.mark.parametrize("graph", [0, 1])
def test_spheres_on_a_mesh(native_lib, graph):
    w = mesh_cloud(600, 0.0, graph_step=graph)
    w.params.rcut_inc = 0.3
    _share(w, 3, 5)
    _both(w, 30)


@pytest.mark.parametrize("spacing", [1.3, 0.9])
def test_polyhedra(native_lib, spacing):
    w = W.polyhedra_lattice(nx=7, ny=7, nz=6, spacing=spacing, seed=3, fused_step=1, fp32_contact_screen=1)
    _share(w, 4, 6)
    _both(w, 5)
