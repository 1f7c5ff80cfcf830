"""Kernels that start while the one before them ends: a run in one call, its
kernels chained, against the same run in calls of one step, each of which ends
with the device idle.  Dimer counts around the eight blocks of eight dimers up to
which the dimer kernel is chained too.

FP64, one collision period and a few steps more: 1e-9, the bound of the other
FP64 comparisons of two runs (their sums differ only in the order of atomics,
about 1e-15 a step)."""
import numpy as np
import pytest

from gpu_helpers import assert_close
from main_gb300 import Engine, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd", [1, 8, 63, 64, 65, 73])
def test_one_call_equals_single_steps(nd):
    cfg = config.workload("c1", seed=3, precision=64, n_dimers=nd)
    states = []
    for chunk in (55, 1):
        e = Engine(cfg)
        e.initial()
        e.prepare()
        for _ in range(0, 55, chunk):
            e.run(chunk)
        states.append(e.download_state())
        e.close()
    assert_close(states[0], states[1], cfg, pos=1e-9, vel=1e-9, flags=1.0, dimer=1e-9)
    assert np.array_equal(states[0]["flag"], states[1]["flag"])
