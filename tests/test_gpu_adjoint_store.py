"""The backward pass reads the step's sums and decisions from the recompute store, joins the gather of a
step with the voxel adjoint of the one before it inside an interval, and keeps its memory and graphs for
a next run of the same lengths.  Any interval gives the same gradient: the stored states are the same
bits, and an interval of one step has no joined launch at all.  Contraction in the two compiled forms
may round differently: 1e-16 of each of some 100 terms per step, 60 steps, with cancellations of up to
1e3 in a sum: 1e-9 of the largest entry.  A second run on the same context repeats the same launches
from the same states: equal bits."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _robots(collide):
    out = []
    for i, dims in enumerate([(1, 1, 1), (5, 4, 3), (9, 7, 6)]):  # one voxel, under and over one warp's links
        rng = np.random.default_rng(i)
        mats = [wl.Material(E=2e5, nu=0.35, cte=0.01),
                wl.Material(E=1e6, nu=0.0, cte=0.01, fail_stress=1e5)]  # some links fail
        out.append(wl.bernoulli_body(rng, dims, 0.85, mats, random_phase=True, temp_vary=True, temp_amplitude=39.0,
                                     enable_collision=collide, enable_expansion=1))
    return out


W = np.array([[-1.0, 0.5, 0.25]] * 3)


@pytest.mark.parametrize("n,collide", [(1, False), (20, False), (60, False), (20, True), (60, True)])
def test_intervals_and_repeated_runs(n, collide):
    robots = _robots(collide)

    def run(b, k):
        b.record(n, k)
        return b.backward(W)

    def fresh(k):
        b = abi.Batch(robots, abi.PRECISION_FP64)
        g = run(b, k)
        b.close()
        return g

    whole = fresh(n)
    assert all(np.all(np.isfinite(g)) and np.abs(g).max() > 0 for g in whole)
    for k in (1, 7):
        for g, w in zip(fresh(k), whole):
            assert np.abs(g - w).max() <= 1e-9 * np.abs(w).max()
    a, b = abi.Batch(robots, abi.PRECISION_FP64), abi.Batch(robots, abi.PRECISION_FP64)
    run(a, 20), run(a, 20)   # kept store and graphs
    run(b, 30), run(b, 60)   # other lengths
    for g, w in zip(run(a, 20), run(b, 20)):
        assert np.array_equal(g, w)
    a.close(), b.close()
