"""The statistics of a move list with more moves in one cell than 16 bits count."""
import numpy as np
import pytest

from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,prm", [(W.SPHERE, [0.5]), (W.SPHEROCYLINDER, [1.0, 0.5])])
@pytest.mark.parametrize("n", [1, 32768, 70001, 140000])
def test_long_move_lists_count_every_move(engine, kind, prm, n):
    from rampack_gb300.packing import MOVE_DTYPE, GpuPacking
    pos = W.lattice((6, 6, 6), (4.0, 4.0, 4.0)) + 0.3
    with GpuPacking(kind, np.array(prm), pos, W.aligned_rotations(len(pos)), W.diag_box(24.0, 24.0, 24.0)) as g:
        g.set_grid((0.0, 0.0, 0.0))
        _, cells, _ = g.grid()
        before = g.stats()
        moves = np.zeros(n, dtype=MOVE_DTYPE)
        moves["particle"] = 17
        moves["domain"] = cells[17]
        moves["uniform"] = 0.5
        moves["rotation"] = np.eye(3).reshape(9)
        codes = g.run_moves(moves)
        after = g.stats()
        d = {k: after[k] - before[k] for k in ("moves", "accepted", "translations", "accepted_translations", "rejected_overlap")}
        assert d == dict(moves=n, accepted=n, translations=n, accepted_translations=n, rejected_overlap=0)
        assert len(set(codes)) == 1
