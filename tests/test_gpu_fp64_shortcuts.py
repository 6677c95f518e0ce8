"""FP64 work decided on the integer pipe in the contact law and the integration,
bit for bit against the oracle's plain formulas: the moment update and its
rolling clip (kr zero and not; spins zero, of either sign, equal, far apart in
magnitude, subnormal), the velocity of a point of a body without spin, the
Euler equations of equal and unequal inertias, and the displacement trigger
across powers of two and near zero."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

FLAGS = dict(fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1)


@pytest.mark.parametrize("kr,inertia", [(0.0, "equal"), (100.0, "equal"), (100.0, "unequal"), (0.0, "mixed")])
def test_spins_and_inertias_bit_exact(native_lib, kr, inertia):
    w = W.spheres_floor(n=3000, side=12.0, seed=71, **FLAGS)
    rng = np.random.default_rng(71)
    vals = np.array([0.0, -0.0, 1.5, -1.5, 1e-70, 3e-65, -2e90, 5e-324])
    for f in ("vrotx", "vroty", "vrotz"):
        pick = rng.integers(0, 4, w.n)
        pick[:40] = rng.integers(0, len(vals) - 2, 40)
        w.particles[f] = vals[pick].copy()
    w.particles["vrotx"][40:60] = 5e-324
    if inertia != "equal":
        k = rng.random(w.n) < (1.0 if inertia == "unequal" else 0.5)
        w.particles["inertiay"] = np.where(k, 1.5 * w.particles["inertiay"], w.particles["inertiay"])
    w.params.config.kr = w.params.config_driver.kr = kr
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(200)
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
    assert_same_list(g.interactions(), o.interactions())
    assert g.rebuild_count() == o.rebuild_count()


@pytest.mark.parametrize("lo", [(0.0, 0.0, 0.0), (-16.0, -15.9, -0.03)])
def test_displacement_trigger_steps(native_lib, lo):
    """The rebuild steps of a box whose coordinates cross zero and powers of two."""
    w = W.spheres_box(n=1500, box=16.0, density=2.0, seed=72, **FLAGS)
    for c, f in enumerate(("rx", "ry", "rz")):
        w.particles[f] = w.particles[f] + lo[c]
    w.params.bounds_lo[:] = list(lo)
    w.params.bounds_hi[:] = [x + 16.0 for x in lo]
    for q, s in enumerate(w.surfaces):
        s["offset"] = lo[q // 2] + (16.0 if q % 2 else 0.0)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(250)
    assert g.rebuild_count() == o.rebuild_count() > 3
    _bits_equal(g.particles(sort_by_id=True), o.particles(sort_by_id=True))
