"""Sphere sweeps with a soft part decide in FP32 where the error bound allows: they must leave the
state of the sweeps that decide every move in FP64, and the total energy must be the oracle's, for
steep and flat potentials, hot and cold, from overlapping starts, odd boxes and few particles."""
import numpy as np
import pytest

import pyoracle as po
from rampack_gb300 import workloads as W

pytestmark = pytest.mark.gpu

WCA, SIC = 1, 2


def start(counts, spacing, jitter, seed):
    rng = np.random.default_rng(seed)
    pos = W.lattice(counts, (spacing,) * 3) + rng.uniform(-jitter, jitter, (int(np.prod(counts)), 3))
    side = np.array(counts) * spacing
    box = W.diag_box(*side)
    box[1], box[5] = 0.05 * side[1], -0.03 * side[2]
    rel = np.mod(pos / side, 1.0)
    rel[rel >= 1.0] = 0.0
    return W.SPHERE, np.array([0.5]), np.ascontiguousarray(rel @ box.reshape(3, 3).T), W.aligned_rotations(len(pos)), box


@pytest.mark.parametrize("kind,eps,sigma,hard,spacing,jitter,temperature", [
    (WCA, 1.0, 1.0, False, 1.1, 0.05, 1.0), (WCA, 1.0, 1.0, False, 0.8, 0.4, 1.0), (WCA, 50.0, 1.0, False, 1.1, 0.3, 0.1),
    (WCA, 1e-3, 1.3, False, 0.9, 0.4, 5.0), (WCA, 2.0, 1.4, True, 1.2, 0.09, 0.7), (SIC, 1.0, 1.0, False, 0.7, 0.3, 0.5),
    (SIC, -2.0, 1.2, False, 0.9, 0.3, 1.0), (SIC, 300.0, 1.5, True, 1.3, 0.1, 1.0)])
@pytest.mark.parametrize("counts", [(6, 7, 5), (13, 9, 11)])
def test_fp32_decisions_leave_the_fp64_state(oracle, engine, kind, eps, sigma, hard, spacing, jitter, temperature, counts):
    from rampack_gb300.packing import GpuPacking
    cfg = start(counts, spacing, jitter, 11)
    states = []
    for fp64_only in (False, True):
        with GpuPacking(*cfg) as g:
            g.set_soft(kind, eps, sigma, hard)
            g.set_temperature(temperature)
            if not fp64_only:
                cpu = po.CpuPacking("oracle", *cfg, threads=1)
                cpu.set_soft(kind, eps, sigma, hard)
                e = cpu.total_energy()
                assert abs(g.total_energy() - e) <= 1e-11 * max(1.0, abs(e))
            out = [g.sweep(0.15, 0.2 * (c % 2), seed=3, counter=c, fp64_only=fp64_only) for c in range(5)]
            assert 0 < sum(s["accepted"] for s in out)
            states.append((g.state(), [(s["moves"], s["accepted"], s["rejected_overlap"], s["rejected_domain"]) for s in out]))
    (a, sa), (b, sb) = states
    assert sa == sb
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
