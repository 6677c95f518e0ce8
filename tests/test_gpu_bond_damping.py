"""The damping coefficient that a bond carries follows what it is made of: after new
inner bond parameters, new bonds and particles of other masses the steps have the
oracle's bits, and a rebuild between two breaks keeps each bond's own."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import pair
from tests.test_gpu_bonds import FAST, assert_same_bonds, assert_same_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [{}, FAST], ids=["plain", "fused"])
def test_bond_damping_follows_its_inputs(native_lib, flags):
    w = W.fragment_blocks(nblocks=2, nx=3, ny=2, nz=2, seed=4,
                          bond=dict(kn=1e4, kt=8e3, damp_rate=0.87, g=0.05), **flags)
    both = pair(w)

    def check():
        assert_same_bonds(*both)
        assert_same_particles(*both)

    for s in both:
        s.first_iteration()
        s.step(60)
    check()
    for s in both:
        s.set_inner_bond_params(dict(kn=7e3, kt=5e3, damp_rate=0.4, g=0.05))
        s.step(40)
    check()
    for s in both:
        p, b = s.particles(), s.bonds()
        p["mass"] = np.ascontiguousarray(p["mass"] * (1.0 + (p["id"] % np.uint64(3)).astype(np.float64)))
        s.set_particles(p)
        s.set_bonds(b)
        s.first_iteration()
        s.step(300)
    check()
