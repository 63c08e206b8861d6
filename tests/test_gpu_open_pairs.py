"""Sweeps of multi-centre bodies in a box so wide that FP32 leaves every pair of neighbours open, more of
them than a warp's queue of undecided pairs holds: all near bodies are then decided in FP64, and each
logged move replays on the CPU oracle."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu

CUBE = np.array([[x, y, z] for x in (-0.3, 0.3) for y in (-0.3, 0.3) for z in (-0.3, 0.3)])
SPHERES = W.polysphere_params(CUBE, 0.5)
SEGMENTS = W.polyspherocylinder_params([(*c, 0.0, 0.0, 0.2, 0.4) for c in CUBE])


@pytest.mark.parametrize("kind,prm,reach", [(W.POLYSPHERE, SPHERES, 0.8), (W.POLYSPHEROCYLINDER, SEGMENTS, 0.9)])
@pytest.mark.parametrize("side", [40.0, 4e5, 1.6e6])
@pytest.mark.parametrize("bulk", [False, True])
@pytest.mark.parametrize("counts", [(3, 3, 3), (3, 4, 4)])    # within what a warp stages there, and beyond it
def test_open_pairs_replay_on_oracle(oracle, engine, kind, prm, reach, side, bulk, counts):
    from rampack_gb300.packing import GpuPacking
    rng = np.random.default_rng(8)
    n, d = int(np.prod(counts)), 2.0 * reach + 0.12
    pos = W.lattice(counts, (d,) * 3) + rng.uniform(-0.05, 0.05, (n, 3)) + 0.37 * side
    cfg = (kind, prm, pos, W.aligned_rotations(n), W.diag_box(side, side, side))
    cpu = po.CpuPacking("oracle", *cfg, threads=1)
    with GpuPacking(*cfg) as g:
        g.set_bulk_staging(bulk)    # the launches of larger systems
        assert g.count_total_overlaps(False) == cpu.count_overlaps(False) == 0
        accepted = 0
        for cycle in range(4):
            st = g.sweep(0.1, 0.1, seed=6, counter=cycle, log=True)
            moves, codes = g.sweep_log()
            want, _ = cpu.replay(moves, g.grid()[2])
            assert np.array_equal(codes, want), (cycle, np.count_nonzero(codes != want))
            accepted += st["accepted"]
        assert accepted > 0
        gp, gr, _ = g.state()
        cp, cr, _ = cpu.state()
        assert np.array_equal(gp, cp) and np.array_equal(gr, cr)
