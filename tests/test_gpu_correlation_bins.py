"""Pair correlations with so many bins that a block's histograms, next to the kernel's static shared memory,
pass the 48 KB that need no opt-in, against the oracle."""
import numpy as np
import pytest

import pyoracle as po
import systems
from test_correlation_oracle import case_desc
from test_gpu_correlation import assert_same, observable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [2816, 2817, 3072, 3242, 3243, 3300, 4096, 4097])
@pytest.mark.parametrize("fn", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("en", [0, 1, 2])
def test_many_bins_match_the_oracle(oracle, engine, en, fn, nb):
    from rampack_gb300.packing import GpuPacking
    cfg = systems.sc_l2()
    case = ("sc_l2", en, 2, (0, 1, 1), fn, 0, "o", 3.0, nb)
    _, d = case_desc(case)
    want = po.OracleCorrelation(d)
    want.add_snapshot(*cfg[2:5])
    with observable(case) as obs, GpuPacking(*cfg) as g:
        obs.add_snapshot(g)
        assert_same(fn, obs.values(), want.values())
