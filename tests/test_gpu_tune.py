"""The autotuner times the schedule that a solve runs: its time per step of the
default variant against the slope of whole solves over their step count, at a
size where stepping directions apart (lattices that fit L2 one at a time)
takes three quarters of stepping them together."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seconds(solid, steps):
    from flow_anizotropy_b200.solver import Params3D, solve3d
    p = Params3D(eps=0.0, lag=steps, min_steps=steps, max_steps=steps, avg_steps=0, precision="fp64", criterion="drift")
    best = 1e9
    for _ in range(3):
        t = time.perf_counter()
        solve3d(solid, 1e-6 * np.eye(3), p)
        best = min(best, time.perf_counter() - t)
    return best


def test_tuned_time_is_a_solves_time(gpu):
    from flow_anizotropy_b200.solver import tune3d
    solid = (np.random.default_rng(2).random((80, 80, 80)) < 0.25).astype(np.uint8)
    ms = tune3d(solid, ndir=3, precision="fp64", nsteps=192)[1][0]
    slope = (_seconds(solid, 1920) - _seconds(solid, 640)) / 1280 * 1e3
    print(f"tuner {ms * 1e3:.1f} us per step, solve {slope * 1e3:.1f}")
    assert abs(ms - slope) < 0.15 * slope
