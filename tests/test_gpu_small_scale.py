"""Rods and bodies of segments in units far smaller than one, where the reference's closest points of two
segments take numerators below 1e-10 for zero, so that its distance is above the geometric one and depends on
which body comes first: moves of sweeps and single moves (the mover first) are the oracle's, and the recount
is the oracle's pair test with the lower index first."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import workloads as W
from test_gpu_pair_filter import rotations

pytestmark = pytest.mark.gpu

ROD = {"rod": (0.01, 0.005), "short_rod": (0.004, 0.005), "thin_rod": (0.03, 0.002), "unit_rod": (0.5, 0.5)}
BENT = {"bent": 0.01, "bent_small": 0.004}
NAMES = [*ROD, *BENT]


def shape(name):
    if name in ROD:
        l, r = ROD[name]
        return W.SPHEROCYLINDER, np.array([l, r]), W.spherocylinder_volume(l, r), l + 2 * r
    s = BENT[name]
    return W.POLYSPHEROCYLINDER, W.polyspherocylinder_params([tuple(s * x for x in c) for c in W.BENT_ROD]), 0.35 * s ** 3, 1.9 * s


def system(name, n, phi, seed):
    rng = np.random.default_rng(seed)
    kind, prm, vol, _ = shape(name)
    side = (n * vol / phi) ** (1.0 / 3.0) * np.array([1.0, 0.9, 1.1])
    box = W.diag_box(*side)
    box[1] = 0.1 * side[1]
    pos = rng.uniform(0.0, 0.999999, (n, 3)) @ box.reshape(3, 3).T
    return (kind, prm, np.ascontiguousarray(pos), rotations(rng, n, None), box), side[0] / n ** (1.0 / 3.0)


@pytest.mark.parametrize("name", NAMES)
def test_recount_takes_the_lower_index_first(oracle, engine, name):
    from rampack_gb300.packing import GpuPacking
    rng = np.random.default_rng(3)
    kind, prm, _, length = shape(name)
    n, side = 400, 60.0 * length
    pos = 30.0 * length + rng.uniform(-1.0, 1.0, (n, 3)) * length
    rot = rotations(rng, n, None)
    body = np.zeros((1, 3)) if name in ROD else BENT[name] * np.array(W.BENT_ROD)[:, :3]
    at = pos[:, None, :] + np.einsum("nij,cj->nci", rot.reshape(n, 3, 3), body)      # the interaction centres
    want = sum(po.pair_overlap("oracle", kind, prm, at[i, a], rot[i], at[j, b], rot[j], a, b)
               for i in range(n) for j in range(i + 1, n) for a in range(len(body)) for b in range(len(body)))
    with GpuPacking(kind, prm, pos, rot, W.diag_box(side, side, side)) as g:
        assert g.count_total_overlaps(False) == want > 1000


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("counting", [False, True])
def test_sweeps_replay_on_oracle(oracle, engine, name, counting):
    from rampack_gb300.packing import GpuPacking
    cfg, unit = system(name, 4000, 0.5 if counting else 0.1, 7)
    cpu = po.CpuPacking("oracle", *cfg, threads=1)
    with GpuPacking(*cfg) as g:
        for q in (cpu, g):
            q.set_counting(counting)
        for cycle in range(6):
            g.sweep(0.3 * unit, 0.5, seed=12, counter=cycle, log=True)
            moves, codes = g.sweep_log()
            want, _ = cpu.replay(moves, g.grid()[2])
            assert np.array_equal(codes, want), np.count_nonzero(codes != want)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("counting", [False, True])
def test_single_moves_replay_on_oracle(oracle, engine, name, counting):
    from rampack_gb300 import _lib
    from rampack_gb300.packing import GpuPacking
    n, m = 3000, 3000
    cfg, unit = system(name, n, 0.5 if counting else 0.1, 11)
    cpu = po.CpuPacking("oracle", *cfg, threads=1)
    rng = np.random.default_rng(4)
    moves = np.zeros(m, dtype=_lib.MOVE_DTYPE)
    moves["particle"] = rng.integers(0, n, m)
    moves["type"], moves["domain"], moves["uniform"] = 2, -1, 0.5
    moves["translation"] = rng.uniform(-0.5, 0.5, (m, 3)) * unit
    moves["rotation"] = rotations(rng, m, 0.3)
    with GpuPacking(*cfg) as g:
        for q in (cpu, g):
            q.set_counting(counting)
        codes, _ = cpu.replay(moves, None)
        got = np.zeros(m, dtype=np.uint8)
        for i, move in enumerate(moves):
            e = g.try_move(int(move["particle"]), 2, move["translation"], move["rotation"])
            got[i] = (1 if e > 0 else (3 if e < 0 else 0)) | (0 if e > 0 else _lib.CODE_ACCEPTED)
            if e <= 0.0:
                g.accept_move()
    assert np.array_equal(got, codes), np.count_nonzero(got != codes)
    assert 0 < np.count_nonzero(got & _lib.CODE_ACCEPTED) < m
