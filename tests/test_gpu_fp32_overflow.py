"""Soft spheres and convex bodies crowded into one cell, more than an FP32 sweep stages: those cells are
swept in FP64 between the others, and the state is the FP64 sweep's."""
import numpy as np
import pytest

from rampack_gb300 import _lib
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def crowded(n, crowd, side, extent, seed):
    rng = np.random.default_rng(seed)
    rel = rng.uniform(0.001, 0.999, (n, 3))
    rel[:crowd] = 0.5 + rng.uniform(-0.5, 0.5, (crowd, 3)) * extent / side
    rot = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    rot *= np.linalg.det(rot)[:, None, None]
    return rel * side, rot.reshape(n, 9), W.diag_box(side, side, side)


@pytest.mark.parametrize("kind,crowd", [(_lib.SHAPE_SPHERE, 900), (_lib.SHAPE_CONVEX, 700)])
def test_crowded_cells_leave_the_fp64_state(engine, kind, crowd):
    from rampack_gb300.packing import GpuPacking
    convex = kind == _lib.SHAPE_CONVEX
    pos, rot, box = crowded(crowd + 3000, crowd, 30.0 if convex else 13.0, 2.0 if convex else 0.9, 3)
    states = []
    for fp64_only in (False, True):
        with GpuPacking(kind, "cuboid 1 1 2; sphere 0.1; sum" if convex else np.array([0.5]), pos, rot, box) as g:
            g.set_cells_per_warp(2)   # spheres: the launches of larger systems
            if not convex:
                g.set_soft(2, 1.0, 1.0, False)
                g.set_temperature(1.0)
            out = [g.sweep(0.2, 0.2, seed=4, counter=c, fp64_only=fp64_only) for c in range(3)]
            states.append((g.state(), [(s["moves"], s["accepted"], s["rejected_overlap"], s["rejected_domain"]) for s in out]))
    (a, sa), (b, sb) = states
    assert sa == sb and 0 < sa[0][1]
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
