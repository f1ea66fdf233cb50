"""The tuners of a batch time what a run of the batch is: their trial time is the
time of a run of as many steps in the chosen shape.  The replicas are uneven, so
that a launch consists of several kernels (one per cluster size) side by side;
one after another they take the sum of their times, several times as long.

Tolerance: the run is timed around its host calls, so it may only be
longer; clocks and the kernels' overlap vary by less than a quarter between runs."""
import numpy as np
import pytest

import femmd_old_gb300 as F
from femmd_old_gb300 import scene as S

pytestmark = pytest.mark.gpu
SIZES = [20000, 12000, 7000, 5000, 3600, 2500, 1800, 1200, 900, 700, 600, 500]


def batch():
    b, systems = F.Batch(0), []
    for k, n in enumerate(SIZES):
        s = F.System(0)
        S.mixed_replica(n, 0.7, 0.5, seed=100 + k).replay(s)
        systems.append(s)
        b.add(s)
    b.run(5)
    return b, systems


def shortest_run(b, systems, start, steps):
    ms = []
    for _ in range(5):
        for s, (x, v) in zip(systems, start):
            s.set_state(x, v)
        b.event_record(0)
        b.run(steps)
        b.event_record(1)
        ms.append(b.event_elapsed_ms(0, 1))
    return min(ms)


@pytest.mark.parametrize("steps", [100, 400])
def test_launch_shape_trial(steps):
    b, systems = batch()
    start = [s.get_state()[:2] for s in systems]
    t = b.autotune(steps)
    for s, (x, v) in zip(systems, start):
        assert np.array_equal(s.get_state()[0], x) and np.array_equal(s.get_state()[1], v)
    assert t["trial_ms"] <= 1.25 * shortest_run(b, systems, start, steps)


def test_list_trial():
    b, systems = batch()
    start = [s.get_state()[:2] for s in systems]
    t = b.autotune_lists(200, skins=(0.3, 0.5), factors=(1.0,))
    assert t["trial_ms"] <= 1.25 * shortest_run(b, systems, start, 200)
