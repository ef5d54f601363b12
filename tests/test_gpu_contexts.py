"""Contexts in one process do not disturb each other: the contact-list rebuild takes as much shared memory
as its context's largest robot needs, and a context with smaller robots may be created at any time."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_a_later_context_with_smaller_robots(precision):
    def batch(cells):
        rng = np.random.default_rng(cells)
        mats = [wl.Material(E=2e5, nu=0.35, cte=0.01)]
        return abi.Batch([wl.bernoulli_body(rng, (cells,) * 3, 0.8, mats, random_phase=True, temp_vary=True, temp_amplitude=39.0,
                                            enable_collision=True)], precision)

    def run(disturb):
        large, small = batch(16), None  # some 2,200 surface voxels, and 56
        large.step(3)
        if disturb:
            small = batch(4)
        large.step(105)  # a graph of 100 steps, and single ones
        pos = large.state()["pos"].copy()
        if small:
            small.step(3)
            small.close()
        large.close()
        return pos

    assert np.array_equal(run(False), run(True))
