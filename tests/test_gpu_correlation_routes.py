"""Radial pair correlations of even and crowded states on both sides of the rule that gives a warp a cell's
points or a point, against the oracle."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import correlation as K
from rampack_gb300 import workloads as W
from test_gpu_correlation import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side", [(300, 15.0), (2000, 15.0), (6000, 40.0), (13000, 44.0), (13000, 24.0)])
@pytest.mark.parametrize("crowded", [0.0, 0.02, 0.4])
@pytest.mark.parametrize("fn", [0, 2])
def test_counts_and_values_match_the_oracle(oracle, engine, n, side, crowded, fn):
    from rampack_gb300.packing import GpuPacking
    rng = np.random.default_rng(n + fn)
    rel = rng.uniform(0.0, 0.999999, (n, 3))
    k = int(n * crowded)
    rel[:k] = 0.97 + rng.uniform(0.0, 1.0, (k, 3)) * (0.5 + 3.0 * crowded) / side     # across the box's corner
    rot = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    rot *= np.linalg.det(rot)[:, None, None]
    pos, rot, box = np.mod(rel, 0.9999999) * side, rot.reshape(n, 9), W.diag_box(side, side, side)
    max_r, nb = 2.0, 40
    want = po.OracleCorrelation(po.pair_desc(function=fn, num_bins=nb, max_r=max_r))
    want.add_snapshot(pos, rot, box)
    obs = (K.PairDensityCorrelation(K.RadialEnumerator(), max_r, nb, print_count=True) if fn == 0 else
           K.PairAveragedCorrelation(K.RadialEnumerator(), K.S220Correlation(), max_r, nb, print_count=True))
    with obs, GpuPacking(W.SPHEROCYLINDER, np.array([0.3, 0.5]), pos, rot, box) as g:
        obs.add_snapshot(g)
        assert_same(fn, obs.values(), want.values())
