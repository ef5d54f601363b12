"""The gradient of a run in which a robot stops: a step that a robot did not take leaves its state as it
was, so its gradient is that of the steps it took, whatever the memory held before.  The arithmetic per
robot is the same in either run (equal operations in equal order; 1e-9 of the largest entry as for
different intervals), and zero exactly where the robot takes no step at all."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu

W = np.array([[-1.0, 0.5, 0.25], [0.75, -0.5, 1.0]])


def _robots(collide):
    out = []
    for i, dims in enumerate([(4, 4, 3), (5, 4, 3)]):
        rng = np.random.default_rng(i)
        mats = [wl.Material(E=1e4 if i == 0 else 2e5, nu=0.35, cte=0.01), wl.Material(E=1e4, nu=0.35, rho=1e6)]
        out.append(wl.bernoulli_body(rng, dims, 0.9, mats[:1], random_phase=True, temp_vary=True, temp_amplitude=39.0,
                                     enable_collision=collide, enable_expansion=1))
        if i == 0:
            out[0].materials = mats
            z, y, x = np.argwhere(out[0].grid > 0)[-1]
            out[0].grid[z, y, x] = 2  # one heavy voxel, that its links do not hold back
    return out


def _batch(robots, speed):
    """The heavy voxel of robot 0 leaves at `speed` (m/s): its links tear (strain above 100) some steps later."""
    b = abi.Batch(robots, abi.PRECISION_FP64)
    s = b.state()
    s["linmom"][b.voxel_offset[1] - 1] = [0.0, 0.0, 1.0 * speed]
    b.set_state(linmom=s["linmom"])
    return b


@pytest.mark.parametrize("collide", [False, True])
@pytest.mark.parametrize("interval", [1, 4, 5, 100])
def test_a_robot_that_tears_in_a_recorded_run(interval, collide):
    robots, speed = _robots(collide), 600.0
    b = _batch(robots, speed)
    taken = 0  # steps that robot 0 takes
    while not b.status()[0]:
        b.step(1)
        taken += 1
        assert taken < 200
    taken -= 1
    assert taken > 1 and not b.status()[1]
    split = b.voxel_offset[1]
    b.close()

    def gradient(n, w, again=False):
        b = _batch(robots, speed)
        b.record(n, interval)
        g = b.backward(w)
        if again:  # the same lengths on the same context: robot 0 takes no step
            b.record(n, interval)
            h = b.backward(w)
            assert all(np.all(x[:split] == 0) for x in h)
            assert all(np.all(np.isfinite(x)) for x in h)
        b.close()
        return g

    whole = gradient(taken + 12, W, again=True)
    short = gradient(taken, W)
    alone = gradient(taken + 12, W * [[0.0], [1.0]])
    for g, s, a in zip(whole, short, alone):
        assert np.all(np.isfinite(g)) and np.abs(s[:split]).max() > 0
        assert np.abs(g[:split] - s[:split]).max() <= 1e-9 * np.abs(s[:split]).max()
        assert np.array_equal(g[split:], a[split:])  # the sound robot's gradient does not know
