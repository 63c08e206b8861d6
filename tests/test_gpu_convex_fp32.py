"""Sweeps of flat convex bodies decide pairs in FP32 where their certificates allow: they must leave the
state of the sweeps that decide every move in FP64, for every primitive and operation, dense and
overlapping starts, sheared boxes, bodies away from their origin, and a few sizes."""
import numpy as np
import pytest

from convex_bodies import BODIES, CIRCUMSPHERE
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MORE = {
    "rounded_box": ("cuboid 1 1 2; sphere 0.1; sum", 1.33),
    "thin_saucer": ("saucer 1 0.05", 1.0),           # a radius of curvature far above the circumsphere
    "displaced": ("cuboid 1 2 1; move 40 0 0; sphere 0.2; move -40 0 0; sum", 1.43),
    "turned_sum": ("segment 2; rot 30 40 50; rectangle 1 0.5; sphere 0.2; sum 3", 1.76),
}
RADII = dict(CIRCUMSPHERE, spherocylinder_sum=1.5, cylinder=1.2, rounded_rectangle=1.3181, tetrahedron=1.0,
             difference=1.3661, sphere=0.5)


@pytest.mark.parametrize("name", sorted(BODIES) + sorted(MORE))
@pytest.mark.parametrize("counts,spacing", [((7, 8, 9), 1.25), ((9, 8, 11), 1.9), ((23, 9, 16), 1.5)])
def test_fp32_decisions_leave_the_fp64_state(engine, name, counts, spacing):
    from rampack_gb300 import _lib
    from rampack_gb300.packing import GpuPacking
    script, circ = MORE[name] if name in MORE else (BODIES[name], RADII[name])
    rng = np.random.default_rng(5)
    n = int(np.prod(counts))
    d = spacing * circ
    side = np.array(counts) * d
    box = W.diag_box(*side)
    box[1], box[5] = 0.04 * side[1], -0.03 * side[2]
    rel = np.mod((W.lattice(counts, (d,) * 3) + rng.uniform(-0.1, 0.1, (n, 3)) * d) / side, 1.0)
    rel[rel >= 1.0] = 0.0
    rot = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    rot *= np.linalg.det(rot)[:, None, None]
    states = []
    for fp64_only in (False, True):
        with GpuPacking(_lib.SHAPE_CONVEX, script, np.ascontiguousarray(rel @ box.reshape(3, 3).T), rot.reshape(n, 9), box) as g:
            out = [g.sweep(0.3 * circ, 0.5, seed=9, counter=c, fp64_only=fp64_only) for c in range(4)]
            states.append((g.state(), [(s["moves"], s["accepted"], s["rejected_overlap"], s["rejected_domain"]) for s in out]))
    (a, sa), (b, sb) = states
    assert sa == sb
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
