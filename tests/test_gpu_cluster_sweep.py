"""Sweeps of small systems in one launch, with neighbourhoods that exceed a warp's share of the shared
memory in some checkerboard phases and not in others (a droplet in a dilute box): every logged move
replays on the CPU oracle and the states are equal."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def droplet(kind, prm, counts, cell, side, seed):
    rng = np.random.default_rng(seed)
    cell, side = np.array(cell), np.array(side)
    pos = W.lattice(counts, cell) + rng.uniform(-0.02, 0.02, (int(np.prod(counts)), 3))
    pos = np.mod(pos + (side - cell * np.array(counts)) / 2, side)
    return kind, prm, np.ascontiguousarray(pos), W.aligned_rotations(len(pos)), W.diag_box(*side)


def crowd(n, crowded, side, seed):
    rng = np.random.default_rng(seed)
    rel = rng.uniform(0.001, 0.999, (n, 3))
    rel[:crowded] = 0.5 + rng.uniform(-0.7, 0.7, (crowded, 3)) / side
    return W.SPHERE, np.array([0.5]), rel * side, W.aligned_rotations(n), W.diag_box(side, side, side)


CHAIN = W.polysphere_params(W.banana_centres(0.6 / (2 * np.sin(np.radians(15))), np.radians(120), 5), 0.5)
CASES = {
    "rods": lambda: droplet(W.SPHEROCYLINDER, np.array([5.0, 0.5]), (6, 6, 10), (1.1, 1.1, 6.2), (70.0, 66.0, 74.0), 1),
    "rods_wide": lambda: droplet(W.SPHEROCYLINDER, np.array([5.0, 0.5]), (10, 10, 6), (1.12, 1.12, 6.3), (70.0, 66.0, 74.0), 2),
    "chains": lambda: droplet(W.POLYSPHERE, CHAIN, (6, 10, 6), (1.9, 1.2, 3.4), (34.0, 31.0, 38.0), 3),
    "bent_rods": lambda: droplet(W.POLYSPHEROCYLINDER, W.polyspherocylinder_params(W.BENT_ROD), (5, 13, 9),
                                 (2.0, 0.62, 0.95), (22.0, 20.0, 24.0), 4),
    "spheres": lambda: crowd(3000, 600, 13.0, 5),
}


def neighbourhoods(cells, dims):
    """The particles in the 27 cells around each occupied cell, and their mean over all cells."""
    occ = np.bincount(cells, minlength=int(np.prod(dims))).reshape(dims[::-1])
    total = np.zeros_like(occ)
    for z in (-1, 0, 1):
        for y in (-1, 0, 1):
            for x in (-1, 0, 1):
                total += np.roll(occ, (z, y, x), (0, 1, 2))
    return total[occ > 0], 27.0 * len(cells) / occ.size


@pytest.mark.parametrize("name", sorted(CASES))
def test_crowded_cells_replay_on_oracle(oracle, engine, name):
    from rampack_gb300.packing import GpuPacking
    cfg = CASES[name]()
    counting = name == "spheres"
    cpu = po.CpuPacking("oracle", *cfg, threads=1)
    with GpuPacking(*cfg) as g:
        dims = g.set_grid((0.0, 0.0, 0.0))["dims"]
        total, mean = neighbourhoods(g.grid()[1], dims)
        assert total.max() > mean + 6.0 * np.sqrt(mean) + 64.0      # beyond a warp's share
        if counting:
            cpu.set_counting(True)
            g.set_counting(True)
        else:
            assert g.count_total_overlaps(False) == 0
        for cycle in range(6):
            st = g.sweep(0.15, 0.0 if counting else 0.1, seed=17, counter=cycle, log=True)
            moves, codes = g.sweep_log()
            want, _ = cpu.replay(moves, g.grid()[2])
            assert np.array_equal(codes, want), (cycle, np.count_nonzero(codes != want))
            assert 0 < st["accepted"] < st["moves"] == len(moves)
        gp, gr, _ = g.state()
        cp, cr, _ = cpu.state()
        assert np.array_equal(gp, cp) and np.array_equal(gr, cr)
        if counting:
            assert g.cached_overlaps() == g.count_total_overlaps(False) == cpu.cached_overlaps()
