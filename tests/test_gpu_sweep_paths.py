"""Small systems' sweeps in one launch and phase by phase (rp_set_cluster_sweep), the latter with cells by
occupancy and in index order: the same states, statistics and logs, and each log replays on the CPU oracle."""
import numpy as np
import pytest

import pyoracle as po
import systems
from test_gpu_cluster_sweep import CASES as CROWDED

pytestmark = pytest.mark.gpu

CASES = ["hs_small", "hs_dense", "sc_l2", "sc_l2_dense", "sc_l5", "poly_banana", "poly_dense", "hs_tiny", "sc_tiny",
         "psc_bent", "psc_tiny"]
PATHS = {"cluster": (True, True), "by_occupancy": (False, True), "by_index": (False, False)}


def sweeps(cfg, path, counting=False, cycles=3, oracle=None, soft=None, **kw):
    from rampack_gb300.packing import GpuPacking
    t, r = (0.1, 0.0) if cfg[0] == 0 else (0.2, 0.2)
    cluster, order = PATHS[path]
    out = []
    with GpuPacking(*cfg) as g:
        g.set_cluster_sweep(cluster)
        g.set_cell_order(order)
        for q in (g, oracle) if oracle else (g,):
            if counting:
                q.set_counting(True)
            if soft:
                q.set_soft(*soft)
        for c in range(cycles):
            st = g.sweep(t, r or kw.get("turn", 0.0), seed=41, counter=c, log=True, rototranslation="turn" in kw)
            assert g.cluster_sweep() == cluster
            moves, codes = g.sweep_log()
            out.append((st["moves"], st["accepted"], st["rejected_overlap"], st["rejected_domain"], moves.tobytes(), codes.tobytes()))
            if oracle:
                want, _ = oracle.replay(moves, g.grid()[2], temperature=1.0)
                assert np.array_equal(codes, want), (c, np.count_nonzero(codes != want))
        out.append(g.cached_overlaps() if counting else 0)
        return [a.tobytes() for a in g.state()], out


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("path", sorted(PATHS))
def test_each_path_replays_on_oracle(oracle, engine, name, path):
    cfg = systems.ALL[name]()
    sweeps(cfg, path, oracle=po.CpuPacking("oracle", *cfg, threads=1))


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("what", ["plain", "counting", "rototranslations"])
def test_the_paths_leave_the_same_state(engine, name, what):
    cfg = systems.ALL[name]()
    if what == "counting":
        cfg = systems.compressed(cfg, 0.97 if "tiny" not in name else 1.0)
    kw = dict(counting=what == "counting", **(dict(turn=0.2) if what == "rototranslations" else {}))
    first = sweeps(cfg, "cluster", **kw)
    for path in ("by_occupancy", "by_index"):
        assert sweeps(cfg, path, **kw) == first, path


@pytest.mark.parametrize("name", sorted(CROWDED))
@pytest.mark.parametrize("path", sorted(PATHS))
def test_crowded_cells_on_each_path(oracle, engine, name, path):
    cfg = CROWDED[name]()
    sweeps(cfg, path, counting=name == "spheres", oracle=po.CpuPacking("oracle", *cfg, threads=1))


@pytest.mark.parametrize("path", sorted(PATHS))
@pytest.mark.parametrize("soft", [(1, 1.0, 1.0, False), (2, 1.0, 1.2, True)])
def test_soft_spheres_on_each_path(oracle, engine, path, soft):
    cfg = systems.ALL["hs_dense"]()
    sweeps(cfg, path, oracle=po.CpuPacking("oracle", *cfg, threads=1), soft=soft)
