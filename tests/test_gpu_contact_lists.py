"""Every surface voxel is listed, whichever thread block its robot's chunk falls to.  Robots of more than
one chunk of 160 surface voxels are binned once per thread block, and the order inside a cell is not the
same in two of them.  Bodies whose actuation brings voxels into contact in the first step, many times
over: after that step FP64 is within 1e-9 voxel sizes of the oracle (one step's rounding is some 1e-16 of
a position; a missed contact moves a voxel by 1e-3), and mixed precision repeats its bits."""

import numpy as np
import pytest

import oracle_bridge as ob
from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _robot(seed, dims):
    rng = np.random.default_rng(seed)
    mats = [wl.Material(E=2e5, nu=0.35, cte=0.01), wl.Material(E=1e6, nu=0.0, cte=0.01)]
    return wl.bernoulli_body(rng, dims, 0.85, mats, random_phase=True, temp_vary=True, temp_amplitude=39.0,
                             enable_collision=True, enable_expansion=1)


# one chunk, two, and several; the smallest body beside a large one
@pytest.mark.parametrize("dims", [[(5, 4, 3)], [(9, 7, 6)], [(5, 4, 3), (9, 7, 6), (14, 13, 12)]])
def test_no_voxel_is_left_out(dims):
    robots = [_robot(i + 1, d) for i, d in enumerate(dims)]
    want = []
    for r in robots:
        o = ob.oracle_sim(r)
        o.step(1)
        want.append(o.voxels()["pos"])
    want = np.concatenate(want)
    first = None
    for _ in range(16):
        b = abi.Batch(robots, abi.PRECISION_FP64)
        b.step(1)
        assert np.count_nonzero(np.abs(b.voxel_aux()["contact"]).sum(1)) > 0
        assert np.max(np.abs(b.state()["pos"] - want)) <= 1e-9 * robots[0].vox_size
        b.close()
        b = abi.Batch(robots, abi.PRECISION_MIXED)
        b.step(20)
        got = b.state()["pos"].copy()
        b.close()
        first = got if first is None else first
        assert np.array_equal(got, first)
