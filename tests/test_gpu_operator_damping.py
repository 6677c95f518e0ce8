"""Contact parameters changed between a list build and the contact operator of a
context with fused_step (dem_set_params, dem_set_multimat), against the oracle bit for
bit: the operator's damping is that of the parameters in place, not of those the list
was built with.  One variant hands the parameters over after the first list, as the
operator graph of a deck does (neighbours first, the contact operator's config last)."""
import numpy as np
import pytest

from exadem_gb300 import system as S
from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

FAST = dict(fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1)


def _operators(s, steps):
    for _ in range(steps):
        s.combined_compute_prolog()
        if s.particle_displ_over():
            s.update_particle_neighbors()
        s.reset_force_moment()
        s.gravity_force()
        s.contact_sphere()
        s.force_to_accel()
        s.combined_compute_epilog()


def _drum(seed, groups=0):
    w = W.spheres_drum(n=1500, seed=seed, **FAST)
    if groups:
        w.particles["group"] = np.random.default_rng(seed).integers(0, groups, w.n).astype(np.uint32)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
        s.step(1500)
        s.update_particle_neighbors()
    assert o.simulation_state()["n_active_interactions"] > 100
    return w, g, o


def _same(g, o):
    _bits_equal(g.particles(), o.particles())
    lg, lo = g.interactions(), o.interactions()
    assert_same_list(lg, lo)
    for k in ("friction", "moment"):
        assert np.array_equal(lg[k], lo[k]), k


@pytest.mark.parametrize("steps", [1, 30])
def test_set_params_before_the_operator(native_lib, steps):
    w, g, o = _drum(71)
    p = w.params
    p.config = S.contact_params(kn=2.5e4, kt=2e4, mu=0.35, damp_rate=0.4)
    p.config_driver = S.contact_params(kn=3e4, kt=2.4e4, mu=0.4, damp_rate=0.5)
    for s in (g, o):
        s.set_params(p)
        _operators(s, steps)
    _same(g, o)


@pytest.mark.parametrize("steps", [1, 30])
def test_set_multimat_before_the_operator(native_lib, steps):
    _, g, o = _drum(72, groups=2)
    a = S.contact_params(kn=1.5e4, kt=1.2e4, mu=0.3, damp_rate=0.5)
    b = S.contact_params(kn=3e4, kt=2.4e4, mu=0.45, damp_rate=0.8)
    d = S.contact_params(kn=2e4, kt=1.6e4, mu=0.4, damp_rate=0.6)
    for s in (g, o):
        s.set_multimat([[a, b], [b, a]], [[d], [d]])
        _operators(s, steps)
    _same(g, o)


def test_parameters_after_the_first_list(native_lib):
    w, g0, o0 = _drum(73)
    w.particles = o0.particles()
    real = S.contact_params(kn=2e4, kt=1.6e4, mu=0.3, damp_rate=0.6)
    none = S.contact_params(kn=0.0, kt=0.0, mu=0.0, damp_rate=0.0)
    w.params.config = w.params.config_driver = none
    g, o = pair(w)
    for s in (g, o):
        s.update_particle_neighbors()
    w.params.config = w.params.config_driver = real
    for s in (g, o):
        s.set_params(w.params)
        s.reset_force_moment()
        s.gravity_force()
        s.contact_sphere()
    _same(g, o)
    for s in (g, o):
        s.force_to_accel()
        _operators(s, 20)
    _same(g, o)
