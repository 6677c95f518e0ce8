"""Particles exchanged with arrays on the device (dem_set_particles and
dem_get_particles, on_device = 1): every field at every alignment a caller's array
can have, absent fields, odd counts; and the operators of a context with fused_step
(their contact law is the fused step's) against the oracle's, dn = 0 included."""
import ctypes as C

import numpy as np
import pytest

from exadem_gb300 import _abi as A
from exadem_gb300 import workloads as W
from exadem_gb300.system import System
from tests.helpers import assert_same_list, pair
from tests.test_gpu_shortcuts import _bits_equal

pytestmark = pytest.mark.gpu

CT = {"id": (C.c_uint64, 8), "type": (C.c_uint32, 4), "group": (C.c_uint32, 4)}


def _device(torch, arrays, shift):
    """The arrays in device memory, field k starting `shift` elements after an aligned address."""
    keep, st = {}, A.Particles()
    st.n = len(arrays["rx"])
    for k, v in arrays.items():
        ct, size = CT.get(k, (C.c_double, 8))
        raw = np.ascontiguousarray(v).view(np.uint8)
        t = torch.zeros(len(raw) + 64, dtype=torch.uint8, device="cuda")
        t[shift * size: shift * size + len(raw)] = torch.from_numpy(raw.copy()).cuda()
        keep[k] = (t, shift * size, len(raw))
        setattr(st, k, C.cast(C.c_void_p(t.data_ptr() + shift * size), C.POINTER(ct)))
    torch.cuda.synchronize()
    return st, keep


@pytest.mark.parametrize("n", [1, 31, 257, 5003])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_device_round_trip(native_lib, n, shift):
    import torch

    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1)
    rng = np.random.default_rng(n)
    arr = {f: rng.uniform(0.1, 9.0, n) for f in A.PARTICLE_FIELDS}
    arr["id"] = rng.permutation(n).astype(np.uint64)
    arr["type"] = rng.integers(0, 5, n).astype(np.uint32)
    arr["group"] = rng.integers(0, 5, n).astype(np.uint32)
    s = System(w.params)
    st, keep = _device(torch, arr, shift)
    s._check(s.b.set_particles(s.h, C.byref(st), 1), "set_particles")
    s.n = n
    back = s.particles(sort_by_id=False)
    for k in arr:
        assert np.array_equal(back[k], arr[k]), k
    out, okeep = _device(torch, {k: np.zeros_like(v) for k, v in arr.items()}, shift)
    s._check(s.b.get_particles(s.h, C.byref(out), 1), "get_particles")
    for k, (t, at, size) in okeep.items():
        raw = t.cpu().numpy()
        assert np.array_equal(raw[at: at + size], np.ascontiguousarray(arr[k]).view(np.uint8)), k
        assert not raw[:at].any() and not raw[at + size:].any(), f"{k}: written outside"


@pytest.mark.parametrize("on_device", [0, 1])
def test_absent_fields_and_radius_bound(native_lib, on_device):
    """Defaults of absent fields, and the list's reach from the largest radius wherever it sits."""
    import torch

    n = 300
    rng = np.random.default_rng(7)
    arr = {f: rng.uniform(1.0, 9.0, n) for f in ("rx", "ry", "rz")}
    arr["radius"] = np.full(n, 0.2)
    arr["radius"][n - 1] = 1.7
    w = W.spheres_box(n=8, box=10.0, density=2.0, seed=1)
    w.particles = dict(W.empty_particles(n), **arr, id=np.arange(n, dtype=np.uint64))
    for f in ("qw", "inertiax", "inertiay", "inertiaz", "mass", "homothety"):
        w.particles[f] = np.ones(n)
    _, o = pair(w)
    s = System(w.params)
    for kw in w.surfaces:
        s.register_surface(**kw)
    st, keep = _device(torch, arr, 0) if on_device else (A.particles_struct(arr, n), None)
    s._check(s.b.set_particles(s.h, C.byref(st), on_device), "set_particles")
    s.n = n
    for q in (s, o):
        q.first_iteration()
    assert_same_list(s.interactions(), o.interactions())
    _bits_equal(s.particles(), o.particles())


@pytest.mark.parametrize("law", ["none", "cohesive"])
def test_operators_of_a_fused_context(native_lib, law):
    flags = dict(fused_step=1, fp32_contact_screen=1, fp32_broad_phase=1)
    if law == "none":
        w = W.spheres_box(n=1500, box=16.0, density=2.0, seed=5, **flags)
        w.particles["rx"][:20] = w.particles["radius"][:20]  # dn = 0 exactly at a wall
    else:
        w = W.spheres_floor(n=2000, side=12.0, seed=5, **flags)
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    assert g.simulation_state()["n_active_interactions"] == o.simulation_state()["n_active_interactions"]
    for _ in range(40):
        for s in (g, o):
            s.combined_compute_prolog()
            if s.particle_displ_over():
                s.update_particle_neighbors()
            s.reset_force_moment()
            s.gravity_force()
            s.contact_sphere()
            s.force_to_accel()
            s.combined_compute_epilog()
    _bits_equal(g.particles(), o.particles())
    assert_same_list(g.interactions(), o.interactions())
    assert g.simulation_state()["n_active_interactions"] == o.simulation_state()["n_active_interactions"]
