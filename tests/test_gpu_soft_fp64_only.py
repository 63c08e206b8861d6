"""Sweeps of a hard core with a soft part, with the FP32 filter and without it: each logged move replays on
the CPU oracle."""
import numpy as np
import pytest

from test_gpu_soft import CASES, make, same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64_only", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_both_arms_replay_on_oracle(oracle, engine, name, fp64_only):
    cfg, cpu, g = make(name)
    t, r = (0.1, 0.0) if cfg[0] == 0 else (0.2, 0.2)
    with g:
        g.set_temperature(1.0)
        for cycle in range(3):
            st = g.sweep(t, r, seed=77, counter=cycle, log=True, fp64_only=fp64_only)
            moves, codes = g.sweep_log()
            want, _ = cpu.replay(moves, g.grid()[2], temperature=1.0)
            assert np.array_equal(codes, want), np.count_nonzero(codes != want)
            assert 0 < st["accepted"] < st["moves"]
        assert same_state(g, cpu)
