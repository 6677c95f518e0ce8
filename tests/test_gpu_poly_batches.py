"""Polyhedron steps launched ahead of the host: the trigger raised at the first step of a
batch, in its middle, in the step after it and not at all, by a vertex displacement and
by a breaking interface, with the call cut into pieces of any length; and the contact
pass's lists by kind of detection at every size of a chunk.  Bit for bit against the
oracle."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

FLAGS = dict(fused_step=1, fp32_broad_phase=1, fp32_contact_screen=1)


@pytest.mark.parametrize("pieces", [[1] * 12, [2, 3, 7, 1, 40], [90], [13, 64, 5]])
@pytest.mark.parametrize("spin", [0.0, 60.0])
def test_pieces_of_a_run(native_lib, pieces, spin):
    w = W.polyhedra_lattice(nx=5, ny=4, nz=4, seed=31, vmax=4.0, **FLAGS)
    rng = np.random.default_rng(31)
    for f in ("vrotx", "vroty", "vrotz"):
        w.particles[f] = rng.uniform(-spin, spin, w.n)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    for k in pieces:
        for s in (g, o):
            s.step(k)
        assert g.rebuild_count() == o.rebuild_count()
    _bits_equal(g.particles(), o.particles())
    assert_same_list(g.interactions(), o.interactions())
    assert g.simulation_state()["n_active_interactions"] == o.simulation_state()["n_active_interactions"]


@pytest.mark.parametrize("pieces", [[1] * 20 + [120], [37, 64, 39]])
def test_breaking_blocks(native_lib, pieces):
    w = W.fragment_blocks(nblocks=3, nx=3, ny=2, nz=2, seed=33, gap=0.01, vz=-4.0, **FLAGS)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    for k in pieces:
        for s in (g, o):
            s.step(k)
        assert g.broken_interface_count() == o.broken_interface_count()
        assert g.rebuild_count() == o.rebuild_count()
    assert g.broken_interface_count() > 0
    _bits_equal(g.particles(), o.particles())
    assert_same_list(g.interactions(), o.interactions())


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (2, 1, 1), (3, 3, 1), (7, 6, 5)])
def test_contact_lists_by_kind(native_lib, nx, ny, nz):
    w = W.polyhedra_lattice(nx=nx, ny=ny, nz=nz, spacing=1.05, seed=34, **FLAGS)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(30)
    _bits_equal(g.particles(), o.particles())
    assert g.simulation_state()["n_active_interactions"] == o.simulation_state()["n_active_interactions"]
