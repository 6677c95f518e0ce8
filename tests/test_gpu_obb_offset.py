"""The pair gate of polyhedra whose box centres lie far from the particles' own origin
(a shape file need not centre its vertices): the list of the FP32 broad phase against
the oracle's for cubes whose boxes are 1e-6 to 1e-2 inside and outside the reach."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair

pytestmark = pytest.mark.gpu


def _turn(q, v):
    u = q[:, 1:]
    uv = np.cross(u, v)
    return v + 2.0 * q[:, :1] * uv + 2.0 * np.cross(u, uv)


@pytest.mark.parametrize("offset", [0.0, 300.0, 1e4, 1e5])
def test_pair_gate_matches_oracle(native_lib, offset):
    w = W.polyhedra_lattice(nx=16, ny=16, nz=2, spacing=4.0, seed=5, fused_step=1, fp32_broad_phase=1,
                            fp32_contact_screen=1)
    rng = np.random.default_rng(int(offset) + 1)
    a = w.particles
    n = len(a["rx"])
    h = n // 2
    away = np.asarray((0.48, -0.6, 0.64)) * offset
    cube = dict(w.shapes[0])
    cube["vertices"] = np.asarray(cube["vertices"]) + away
    cube["obb"] = dict(cube["obb"], center=tuple(np.asarray(cube["obb"]["center"]) + away))
    w.shapes = [cube]
    a["type"][:] = 0
    a["homothety"] = np.ones(n)
    q = rng.standard_normal((h, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    body = np.stack([np.arange(h) % 16, np.arange(h) // 16, np.zeros(h)], 1) * 6.0
    reach = 1.0 + 2.0 * float(cube["radius"]) + float(w.params.rcut_inc)  # edge, two radii, skin
    axis = np.eye(3)[rng.integers(0, 3, h)]
    gap = reach + rng.choice((-1.0, 1.0), h) * 10.0 ** rng.uniform(-6.0, -2.0, h)
    other = body + _turn(q, axis * gap[:, None])
    # the second of a pair has the first one's axes, turned by a half turn about one of
    # them: its origin then lies 2 |away| from the first one's
    half = np.zeros((h, 4))
    half[np.arange(h), 1 + rng.integers(0, 3, h)] = 1.0
    q2 = np.concatenate([(q[:, :1] * half[:, :1] - np.sum(q[:, 1:] * half[:, 1:], 1, keepdims=True)),
                         q[:, :1] * half[:, 1:] + half[:, :1] * q[:, 1:] + np.cross(q[:, 1:], half[:, 1:])], 1)
    pos = np.concatenate([body - _turn(q, np.tile(away, (h, 1))), other - _turn(q2, np.tile(away, (h, 1)))])
    for k, f in enumerate(("rx", "ry", "rz")):
        a[f] = np.ascontiguousarray(pos[:, k])
    for k, f in enumerate(("qw", "qx", "qy", "qz")):
        a[f] = np.ascontiguousarray(np.concatenate([q, q2])[:, k])
    a["radius"] = np.full(n, 1.0 + offset)
    a["id"] = np.arange(n, dtype=np.uint64)
    ext = 2.0 * offset + 200.0
    w.params.bounds_lo[:] = (-ext,) * 3
    w.params.bounds_hi[:] = (ext,) * 3
    w.surfaces, w.cylinders = [], []
    g, o = pair(w)
    for s in (g, o):
        s.update_particle_neighbors()
    lst = o.interactions()
    pairs = len(np.unique(np.stack([lst["owner_id"], lst["partner_id"]]), axis=1).T)
    assert h // 4 < pairs < 3 * h // 4
    assert_same_list(g.interactions(), lst)
