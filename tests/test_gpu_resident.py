"""Many mixed-precision steps in one launch (robots held in the shared memory of a cluster of
CTAs) against the same steps pass by pass: vx3g_autotune advances a batch by timing the passes
of single steps, vx3g_step takes the launch of many steps where the batch allows it.  The two
run the same arithmetic with every rounding spelled out, so everything they leave behind is
equal bit for bit."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _all(b):
    out = dict(b.state(), time=b.time(), status=b.status(), com=b.com(), **b.links())
    aux = b.voxel_aux()
    return dict(out, tempe=aux["tempe"], flags=aux["flags"])


def _same(robots, steps, before=None):
    got = []
    for passes in (True, False):
        b = abi.Batch(robots, abi.PRECISION_MIXED)
        if before:
            before(b)
        if passes:
            b.autotune(sum(steps))
        else:
            for n in steps:
                b.step(n)
        assert b.steps_taken() == sum(steps)
        got.append(_all(b))
        b.close()
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k], equal_nan=True), k
    return got[0]


def _body(rng, dims, fill=0.75, mats=3, **kw):
    m = [wl.Material(E=float(10 ** rng.uniform(5, 7)), nu=0.35, rho=float(rng.uniform(500, 2000)), cte=0.01)
         for _ in range(mats)]
    kw = dict(dict(random_phase=True, temp_vary=True, temp_amplitude=39.0), **kw)
    return wl.bernoulli_body(rng, dims, fill, m, **kw)


# voxels per robot around the edges of a CTA (96 voxels while SMs are idle), of a warp and of
# the largest cluster
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (31, 1, 1), (4, 8, 3), (8, 4, 4), (129, 1, 1), (8, 8, 6), (12, 12, 6),
                                  (11, 13, 17), (16, 16, 16)])
def test_one_robot(dims):
    rng = np.random.default_rng(sum(dims))
    robot = _body(rng, dims, fill=1.0, z_offset=1)
    _same([robot], [1, 2, 37, 60])


@pytest.mark.parametrize("count,lo,hi", [(3, 2, 4), (40, 1, 3), (400, 2, 5), (7, 9, 12), (700, 5, 9)])
def test_batches(count, lo, hi):
    """Bundles of many small robots, several cluster sizes in one batch, and more than one launch."""
    rng = np.random.default_rng(count)
    robots = [_body(rng, tuple(int(x) for x in rng.integers(lo, hi + 1, size=3)), z_offset=i % 2, slow_damping=0.01 * (i % 3))
              for i in range(count)]
    _same(robots, [270])


def test_materials():
    """Fixed voxels, late expansion, failing links, a plastic curve, static expansion, no floor, and
    per-voxel moduli (a link material of its own for every link)."""
    rng = np.random.default_rng(4)
    def fixed(k):
        return wl.Material(E=1e6, nu=0.3, cte=0.01, fixed=k)
    robots = [
        wl.bernoulli_body(rng, (6, 5, 4), 0.9, [fixed(0), fixed(1)], random_phase=True, temp_vary=True, temp_amplitude=39.0),
        wl.bernoulli_body(rng, (5, 5, 5), 0.9, [wl.Material(E=1e6, cte=0.01, thermal_on_after=0.002), wl.Material(E=2e6, cte=0.01)],
                          random_phase=True, temp_vary=True, temp_amplitude=-39.0, enable_expansion=1),
        wl.bernoulli_body(rng, (6, 4, 4), 0.9, [wl.Material(E=1e6, cte=0.01, fail_stress=2e4)], random_phase=True, temp_vary=True,
                          temp_amplitude=39.0, z_offset=2),
        wl.bernoulli_body(rng, (5, 4, 6), 0.9, [wl.Material(E=1e6, nu=0.2, cte=0.01, model=2, plastic_mod=1e5, yield_stress=1e4)],
                          random_phase=True, temp_vary=True, temp_amplitude=39.0),
        wl.bernoulli_body(rng, (4, 4, 4), 0.9, [wl.Material(E=1e6, cte=0.01), wl.Material(E=1e5)], temp_enabled=True, temp_amplitude=10.0,
                          floor=False),
        wl.solid_block(6, drop_cells=1),
    ]
    grad = wl.c4_differentiable(seed=3)[0]
    out = _same(robots + [grad], [130])
    assert np.any(out["small"] & 1 == 0)  # large-angle links among them


def test_a_robot_that_diverges_stops_alone():
    rng = np.random.default_rng(9)
    robots = [_body(rng, (6, 6, 6), z_offset=1) for _ in range(5)]

    def tear(b):
        s = b.state()
        v = b.voxel_offset[2]
        s["pos"][v] += 50.0  # a voxel far away: its links' strain passes 100
        b.set_state(pos=s["pos"])
        b.stop_robot(4)

    out = _same(robots, [90], before=tear)
    assert list(out["status"] != 0) == [False, False, True, False, True]


# either side of the rule that takes such a batch to the one launch: robots of a whole SM per CTA, as many
# as run at once, and twice that (a second wave, slower than the passes)
@pytest.mark.parametrize("count,dims", [(8, (16, 16, 16)), (30, (13, 13, 13))])
def test_large_robots(count, dims):
    rng = np.random.default_rng(count)
    _same([_body(rng, dims, fill=1.0) for _ in range(count)], [3, 40])
