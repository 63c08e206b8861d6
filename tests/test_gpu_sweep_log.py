"""The logged translation of a rotation is zero with a positive sign, for every shape and path."""
import numpy as np
import pytest

import systems
from rampack_gb300 import _lib
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {n: systems.ALL[n] for n in ("hs_small", "sc_l2", "poly_banana", "psc_bent")}
CASES["convex"] = lambda: (_lib.SHAPE_CONVEX, W.ROUNDED_BOX, W.lattice((6, 7, 8), (3.0,) * 3), W.aligned_rotations(336),
                           W.diag_box(18.0, 21.0, 24.0))


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("bulk", [False, True])
@pytest.mark.parametrize("counting", [False, True])
def test_rotations_log_positive_zeros(engine, name, bulk, counting):
    from rampack_gb300.packing import GpuPacking
    with GpuPacking(*CASES[name]()) as g:
        g.set_bulk_staging(bulk)
        g.set_counting(counting)
        g.sweep(0.1, 0.2, seed=5, counter=0, log=True)
        moves, _ = g.sweep_log()
    t = moves["translation"][moves["type"] == 1]
    assert len(t) and not t.any() and not np.signbit(t).any()
    assert np.abs(moves["translation"][moves["type"] == 0]).max() > 0
