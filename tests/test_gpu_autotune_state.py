"""What dem_autotune leaves behind: after a trial that fails, the context as it was; after
a success, the rule that places the integration's multiplies by particle count, unless
a trial beat what it gives."""
import ctypes as C

import numpy as np
import pytest

from exadem_gb300 import workloads as W
from exadem_gb300 import DemError
from tests.helpers import assert_same_list
from tests.test_gpu_shortcuts import _bits_equal
from tests.test_gpu_sphere_lists import _cloud

pytestmark = pytest.mark.gpu

FAST = dict(fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1)
MANY = 20011  # above 128 particles an SM


def _mode(s):
    m = C.c_int(-1)
    s._check(s.b.selftest_integration_mode(s.h, C.byref(m)), "integration_mode")
    return m.value


def _cube(n):
    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1, **FAST)
    side = int(np.ceil(n ** (1 / 3)))
    a = W.empty_particles(n)
    k = np.arange(n)
    for d, f in enumerate(("rx", "ry", "rz")):
        a[f] = (k // side ** d % side + 0.5) * 1.1
    a["radius"] = np.full(n, 0.5)
    for f in ("mass", "qw", "homothety", "inertiax", "inertiay", "inertiaz"):
        a[f] = np.ones(n)
    a["id"] = k.astype(np.uint64)
    w.particles = a
    w.params.bounds_hi[:] = [side * 1.1] * 3
    w.surfaces = []
    return w


@pytest.mark.parametrize("graph", [0, 1])
def test_failed_trial(native_lib, graph):
    w = _cloud(60, 2.7, (1, 1, 1), 4)  # three cells along each axis: three times the skin is too wide
    w.params.graph_step = graph
    a, b = w.build(), w.build()
    for s in (a, b):
        s.first_iteration()
        s.step(20)
    assert _mode(b) == 0
    with pytest.raises(DemError, match="at least 3 cells"):
        b.autotune(steps_per_trial=1, skin_policy=2)
    assert _mode(b) == 0 and b.mul_mode() == a.mul_mode() == 2
    assert a.rebuild_count() == b.rebuild_count()
    assert_same_list(a.interactions(), b.interactions())
    for s in (a, b):
        s.step(60)
    assert a.rebuild_count() == b.rebuild_count()
    assert_same_list(a.interactions(), b.interactions())
    _bits_equal(a.particles(), b.particles())


def test_rule_by_count(native_lib):
    s = _cube(1000).build()
    assert _mode(s) == 0
    s.first_iteration()
    r = s.autotune(steps_per_trial=2, skin_policy=0)
    assert (_mode(s) & 3) == (r["mul_mode"] & 3)
    tuned = s.mul_mode()
    s.set_params(_cube(MANY).params)
    s.set_particles(_cube(MANY).particles)
    assert _mode(s) == (2 if r["mul_mode"] == 0 else tuned)
    s.close()
    s = _cube(MANY).build()
    assert _mode(s) == 2
    s.set_mul_mode(1)
    assert _mode(s) == 1
    s.close()
