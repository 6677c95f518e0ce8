"""The candidate records of the FP32 sphere list build: only the contexts that use them
hold any, and the lists are the oracle's whatever fits: all candidates, those of some
spheres, mesh candidates but not particles, particles but not mesh candidates."""
import ctypes as C

import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair
from tests.test_gpu_mesh_lists import _cloud as mesh_cloud
from tests.test_gpu_shortcuts import _bits_equal
from tests.test_gpu_sphere_lists import _cloud as sphere_cloud

pytestmark = pytest.mark.gpu

FAST = dict(fused_step=1, fp32_contact_screen=1)


def _records(s, budget=0):
    out = (C.c_uint32 * 2)()
    s._check(s.b.selftest_records(s.h, budget, out), "records")
    return tuple(out)


@pytest.mark.parametrize("fp32,cells,want", [(1, 0, (16, 0)), (1, 1, (0, 0)), (0, 0, (0, 0))])
def test_only_the_build_that_uses_them(native_lib, fp32, cells, want):
    s = W.spheres_box(n=500, box=12.0, density=2.0, seed=2, fp32_broad_phase=fp32, graph_step=1, **FAST).build()
    assert _records(s) == (0, 0)
    s.set_sphere_cell_broad_phase(cells)
    s.first_iteration()
    s.step(3)
    assert _records(s) == want
    s.set_sphere_cell_broad_phase(0)  # the records appear before the graph is captured
    s.step(3)
    assert _records(s) == ((16, 0) if fp32 else (0, 0))
    s.close()


def test_polyhedra_hold_none(native_lib):
    s = W.polyhedra_lattice(nx=4, ny=4, nz=3, fp32_broad_phase=1, **FAST).build()
    s.first_iteration()
    s.step(3)
    assert _records(s) == (0, 0)
    s.close()


def _run(w, budget, want):
    g, o = pair(w)
    if budget:
        _records(g, budget)
    for s in (g, o):
        s.first_iteration()
    assert _records(g) == want
    lst = o.interactions()
    assert_same_list(g.interactions(), lst)
    for s in (g, o):
        s.step(60)
    assert g.rebuild_count() == o.rebuild_count()
    assert_same_list(g.interactions(), o.interactions())
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
    return lst


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("budget,want", [(0, (16, 0)), (1, (4, 0))])
def test_spheres(native_lib, budget, want, graph):
    w = sphere_cloud(700, 6.0, (1, 0, 1), 11, 0, 0.0, 0.3)
    w.params.graph_step = graph
    lst = _run(w, budget, want)
    held = np.unique(lst["owner_id"], return_counts=True)[1]
    assert (held > want[0]).any() and (held <= want[0]).any()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("budget,want", [(0, (16, 48)), (600 * 256, (16, 0)), (1, (4, 0))])
def test_spheres_on_a_mesh(native_lib, budget, want, graph):
    w = mesh_cloud(600, 0.0, fp32_broad_phase=1, graph_step=graph)
    w.params.rcut_inc = 0.15
    lst = _run(w, budget, want)
    ids = w.particles["id"].astype(np.int64)
    mesh = np.isin(lst["type"], (7, 8, 9))
    on_mesh = np.bincount(lst["owner_id"][mesh].astype(np.int64), minlength=len(ids))
    others = np.bincount(lst["owner_id"][~mesh].astype(np.int64), minlength=len(ids))
    fits, long = on_mesh <= want[1], others > want[0]
    assert (~fits).any() and (fits & ~long & (on_mesh + others > 0)).any()
    assert (fits & long).any()  # too many particles alone
    assert (~fits & long).any() and (~fits & ~long).any()
