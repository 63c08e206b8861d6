"""The FP32 segment test and the recount on random states with overlaps against the CPU oracle:
short and long rods, parallel, nearly parallel and random axes, boxes two cells across, cells with
one particle and with many, and walls; every count must equal the oracle's."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rotations(rng, n, tilt):
    q = rng.normal(size=(n, 4)) if tilt is None else np.c_[np.ones(n), rng.normal(size=(n, 3)) * tilt]
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    return np.ascontiguousarray(np.stack([
        1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z), 1 - 2 * (x * x + z * z),
        2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1))


def counts(kind, prm, pos, rot, box, walls=0):
    from rampack_gb300.packing import GpuPacking
    cpu = po.CpuPacking("oracle", kind, prm, pos, rot, box, threads=4)
    with GpuPacking(kind, prm, pos, rot, box) as g:
        if walls:
            cpu.set_walls(walls)
            g.set_walls(walls)
        got = g.count_total_overlaps(False), g.count_total_overlaps(True)
        assert got == (cpu.count_overlaps(False), cpu.count_overlaps(True))
        g.set_grid((0.31, 0.77, 0.13))
        assert g.count_total_overlaps(False) == got[0]
    return got[0]


@pytest.mark.parametrize("length", [0.02, 0.7, 2.0, 9.0])
@pytest.mark.parametrize("tilt", [0.0, 1e-6, 1e-4, 0.05, None])
def test_rod_counts(oracle, engine, length, tilt):
    rng = np.random.default_rng(int(1000 * length) + 7)
    side = 2.6 * (length + 1.0)
    box = W.diag_box(side, 1.2 * side, 2.1 * side)
    n = int(0.5 * box[0] * box[4] * box[8] / W.spherocylinder_volume(length, 0.5))
    pos = rng.uniform(0.0, 1.0, (n, 3)) * box[[0, 4, 8]]
    # a lattice share: exact contacts at 1 - and 1 + 1e-7 diameters along the axis and across it
    k = min(n // 2, 40)
    pos[1:2 * k:2] = pos[0:2 * k:2] + np.array([1.0 + 1e-7, 0.0, 0.0]) * rng.choice([1.0, 1.0 - 4e-7], (k, 1))
    pos = np.mod(pos, box[[0, 4, 8]] * (1 - 1e-12))
    assert counts(W.SPHEROCYLINDER, np.array([length, 0.5]), pos, rotations(rng, n, tilt), box) > 0


@pytest.mark.parametrize("n,side", [(1, 4.0), (2, 4.0), (33, 4.2), (513, 6.5), (900, 4.3), (2000, 30.0)])
@pytest.mark.parametrize("walls", [0, 5])
def test_sphere_counts(oracle, engine, n, side, walls):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * side * 0.999999
    counts(W.SPHERE, np.array([0.5]), pos, W.aligned_rotations(n), W.diag_box(side, side, side), walls)


@pytest.mark.parametrize("n", [2, 65, 400])
def test_clustered_cells(oracle, engine, n):
    # one crowded corner of a dilute box: a cell far fuller than a staging tile
    rng = np.random.default_rng(n + 1)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * 3.0 + 1.0
    box = W.diag_box(200.0, 180.0, 220.0)
    counts(W.SPHEROCYLINDER, np.array([2.0, 0.5]), pos, rotations(rng, n, None), box)
    counts(W.SPHERE, np.array([0.5]), pos, W.aligned_rotations(n), box)


@pytest.mark.parametrize("walls", [0, 2])
def test_multi_centre_counts(oracle, engine, walls):
    rng = np.random.default_rng(12)
    box = W.diag_box(9.0, 8.0, 10.0)
    pos = rng.uniform(0.0, 1.0, (300, 3)) * box[[0, 4, 8]] * 0.999999
    rot = rotations(rng, 300, None)
    assert counts(W.POLYSPHEROCYLINDER, W.polyspherocylinder_params(W.BENT_ROD), pos, rot, box, walls) > 0
    chain = W.polysphere_params(W.banana_centres(1.16, 2.0, 5), 0.5)
    assert counts(W.POLYSPHERE, chain, pos, rot, box, walls) > 0


@pytest.mark.parametrize("counting", [False, True])
def test_unequal_segments_replay(oracle, engine, counting):
    """Sweeps of bodies whose segments differ in length and radius (one a sphere), from an aligned
    lattice on: every logged move replays on the oracle, and so do the counts of random states."""
    from rampack_gb300.packing import GpuPacking
    data = ((-0.4, 0.0, 0.0, 0.3, 0.0, 0.2, 0.25), (0.3, 0.0, 0.1, 0.0, 0.0, 0.0, 0.35), (0.0, 0.3, 0.0, 0.0, 0.5, 0.0, 0.15))
    prm = W.polyspherocylinder_params(data)
    pos = W.lattice((5, 6, 7), (1.75, 1.6, 1.2))
    box = W.diag_box(8.75, 9.6, 8.4)
    rot = W.aligned_rotations(len(pos))
    if counting:
        rng = np.random.default_rng(3)
        rot = rotations(rng, len(pos), None)
        assert counts(W.POLYSPHEROCYLINDER, prm, pos, rot, box) > 0
    cpu = po.CpuPacking("oracle", W.POLYSPHEROCYLINDER, prm, pos, rot, box, threads=1)
    with GpuPacking(W.POLYSPHEROCYLINDER, prm, pos, rot, box) as g:
        if counting:
            cpu.set_counting(True)
            g.set_counting(True)
        for cycle in range(4):
            st = g.sweep(0.2, 0.4, seed=5, counter=cycle, log=True)
            moves, codes = g.sweep_log()
            want, _ = cpu.replay(moves, g.grid()[2])
            assert np.array_equal(codes, want), (cycle, np.count_nonzero(codes != want))
            assert 0 < st["accepted"] < st["moves"]
        gp, gr, _ = g.state()
        cp, cr, _ = cpu.state()
        assert np.array_equal(gp, cp) and np.array_equal(gr, cr)
