"""The pair gate of polyhedra (boxes of cubes are aligned with the world whatever the
cubes' orientation, so half of its axes compare values of the tolerance's size): the
list of the FP32 broad phase against the oracle's for cubes at all offsets about the
reach of the enlarged boxes, boxes that touch in a face, an edge or a corner, scaled
shapes and quaternions off unit norm."""
import numpy as np
import pytest

from exadem_gb300 import workloads as W
from tests.helpers import assert_same_list, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,turned,homothety,norm", [
    (1, 0.0, 0.0, 0.0), (2, 1e-9, 0.0, 0.0), (3, 1.0, 0.0, 0.0), (4, 0.5, 0.3, 0.02)])
def test_pair_gate_matches_oracle(native_lib, seed, turned, homothety, norm):
    w = W.polyhedra_lattice(nx=24, ny=24, nz=2, spacing=4.0, seed=seed, fused_step=1, fp32_broad_phase=1,
                            fp32_contact_screen=1)
    rng = np.random.default_rng(100 + seed)
    a = w.particles
    n = len(a["rx"])
    h = n // 2  # particle k of the upper layer sits about its partner in the lower one
    order = np.argsort(a["rz"], kind="stable")
    low, up = order[:h], order[h:]
    a["type"][:] = 0  # cubes
    q = np.zeros((n, 4))
    q[:, 0] = 1.0
    q[:, 1:] = turned * rng.standard_normal((n, 3))
    q /= np.linalg.norm(q, axis=1)[:, None]
    q *= 1.0 + norm * rng.uniform(-1.0, 1.0, (n, 1))
    for k, f in enumerate(("qw", "qx", "qy", "qz")):
        a[f] = np.ascontiguousarray(q[:, k])
    a["homothety"] = 1.0 + homothety * rng.uniform(-1.0, 1.0, n)
    reach = 1.0 + 0.02 + float(w.params.rcut_inc)  # edge, two radii, skin
    out = rng.uniform(-1.0, 1.0, (h, 3))
    for axes in range(3):  # a face, an edge or a corner at the reach
        pick = rng.random(h) < (1.0, 0.5, 0.3)[axes]
        sign = rng.choice((-1.0, 1.0), h)
        eps = sign * 10.0 ** rng.uniform(-12.0, -1.0, h)
        out[pick, axes] = (rng.choice((-1.0, 1.0), h) * (reach + eps))[pick]
    out = np.take_along_axis(out, rng.permuted(np.tile(np.arange(3), (h, 1)), axis=1), axis=1)
    for k, f in enumerate(("rx", "ry", "rz")):
        a[f][up] = a[f][low] + out[:, k]
    g, o = pair(w)
    for s in (g, o):
        s.first_iteration()
    lg, lo = g.interactions(), o.interactions()
    assert len(lo["owner_id"]) > 0
    assert_same_list(lg, lo)
