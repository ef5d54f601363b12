"""The FP64 passes decide branches, and form the temperature, from cheaper quantities wherever
those are clear of the decision, and from the reference's expressions elsewhere.  Against the
oracle (the reference's arithmetic in C): positions within 1e-9 voxel sizes.  The only other
difference between the two is CUDA's sine, cosine and arc cosine (1-2 ulp) against the C
library's; over 150 steps an error of 2e-16 grows by less than 1e4 on these bodies, 2e-12 of a
position of a few voxel sizes.  The temperatures, stored in 32 bits, are equal."""

import numpy as np
import pytest

import oracle_bridge as ob
from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _robot(dims, phase_scale=1.0, amplitude=39.0, **kw):
    rng = np.random.default_rng(sum(dims))
    mats = [wl.Material(E=float(10 ** rng.uniform(5, 7)), nu=0.35, cte=0.01) for _ in range(3)]
    r = wl.bernoulli_body(rng, dims, 0.8, mats, random_phase=True, temp_vary=True, temp_amplitude=amplitude, **kw)
    r.phase = (r.phase - 0.5) * phase_scale
    return r


# one voxel to several blocks; phases beyond the two cycles that the voxel table covers; a negative
# amplitude; expansion on; floor off; standing on the floor and dropped on it
@pytest.mark.parametrize("kw", [dict(dims=(1, 1, 1)), dict(dims=(33, 1, 1)), dict(dims=(7, 5, 6)),
                                dict(dims=(7, 6, 5), phase_scale=9.0), dict(dims=(5, 6, 7), amplitude=-39.0),
                                dict(dims=(6, 6, 6), enable_expansion=1), dict(dims=(6, 7, 6), floor=False),
                                dict(dims=(7, 7, 6), z_offset=1, slow_damping=0.02), dict(dims=(12, 12, 11))])
def test_against_the_oracle(kw):
    robot = _robot(**kw)
    b = abi.Batch([robot], abi.PRECISION_FP64)
    o = ob.oracle_sim(robot)
    b.step(150)
    o.step(150)
    want = o.voxels()
    assert np.max(np.abs(b.state()["pos"] - want["pos"])) <= 1e-9 * robot.vox_size
    assert np.array_equal(b.voxel_aux()["tempe"], want["tempe"])
    b.close()
