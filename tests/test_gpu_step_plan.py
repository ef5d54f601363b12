"""Which way a batch is stepped, as vx3g_step_plan tells it: the other tests of the many-step kernel compare
it with the passes, and here is asserted that it is what runs, in clusters of the sizes that the robots
should take, and that the batches it does not handle keep the passes."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl
import test_gpu_resident as resident
import test_gpu_resident_divergence as divergence

pytestmark = pytest.mark.gpu


def _plan(robots, precision=abi.PRECISION_MIXED):
    b = abi.Batch(robots, precision)
    p = b.step_plan()
    b.close()
    return p


# 96 voxels per thread block while SMs are idle (up to 128 rather than one block more), at most eight
SIZES = [((1, 1, 1), 1), ((2, 1, 1), 1), ((31, 1, 1), 1), ((4, 8, 3), 1), ((8, 4, 4), 1), ((129, 1, 1), 2), ((8, 8, 6), 3),
         ((12, 12, 6), 7), ((10, 10, 10), 8), ((16, 16, 16), 8)]


@pytest.mark.parametrize("dims,size", SIZES)
def test_one_robot(dims, size):
    b = abi.Batch([resident._body(np.random.default_rng(1), dims, fill=1.0)], abi.PRECISION_MIXED)
    if b.nv <= 1000:
        assert 1 <= b.step_plan()["many_from"] < 12  # the rule takes it, for more than a few steps
    b.choose_steps("many")
    p = b.step_plan()
    assert p["many_from"] == 1 and p["most"] >= 100 and p["launches"] == 1 and p["clusters"] == {size: 1}
    b.choose_steps("passes")
    assert b.step_plan()["many_from"] == 0
    b.close()


CLUSTERS = [{1: 1}, {1: 5}, {1: 300}, {2: 3}, {8: 2}]


@pytest.mark.parametrize("form", range(len(divergence.FORMS)))
def test_forms_of_the_divergence_test(form):
    count, dims = divergence.FORMS[form]
    b = abi.Batch([divergence._robot(i, dims) for i in range(count)], abi.PRECISION_MIXED)
    b.choose_steps("many")
    assert b.step_plan()["clusters"] == CLUSTERS[form]
    b.close()


def _mixed_batch(count, lo, hi):
    rng = np.random.default_rng(count)
    return [resident._body(rng, tuple(int(x) for x in rng.integers(lo, hi + 1, size=3)), z_offset=i % 2, slow_damping=0.01 * (i % 3))
            for i in range(count)]


BATCHES = [(3, 2, 4), (40, 1, 3), (400, 2, 5), (7, 9, 12), (30, 11, 13), (700, 5, 9)]


@pytest.mark.parametrize("count,lo,hi", BATCHES)
def test_both_ways_leave_the_same(count, lo, hi):
    """Whatever the rule decides: bundles, several cluster sizes side by side, several waves, and a switch
    between the two ways at odd and even steps."""
    robots, got = _mixed_batch(count, lo, hi), []
    for ways in (["passes"], ["many"], ["many", "passes"]):
        b = abi.Batch(robots, abi.PRECISION_MIXED)
        for i, n in enumerate([1, 2, 37, 60, 13, 120]):
            b.choose_steps(ways[i % len(ways)])
            assert (b.step_plan()["many_from"] > 0) == (ways[i % len(ways)] == "many")
            b.step(n)
        if ways == ["many"]:
            p = b.step_plan()
            assert p["launches"] == len(p["clusters"]) >= (2 if lo >= 9 else 1)
        got.append(resident._all(b))
        b.close()
    for other in got[1:]:
        for k in got[0]:
            assert np.array_equal(got[0][k], other[k], equal_nan=True), k


def test_calls_of_few_and_of_many_steps():
    """A call goes by the passes up to the plan's number of steps, and in launches of equal length above the
    most of one; graphs are captured where a chunk of theirs can still come to run."""
    rng = np.random.default_rng(6)
    robots = [resident._body(rng, (7, 6, 5)) for _ in range(5)]
    got = []
    for chunk in (100, 2, -1):
        b = abi.Batch(robots, abi.PRECISION_MIXED, graph_chunk=chunk)
        b.prepare_graphs()
        if chunk > 0:
            k = b.step_plan()["many_from"]
            assert k > 2
        else:  # no graphs: the kernels of every step, one by one
            assert b.step_plan()["many_from"] == 0
        for n in (1, k - 1, k, k + 1, 256, 257, 513, 2):
            b.step(n)
        got.append(resident._all(b))
        b.choose_steps("passes")
        b.prepare_graphs()
        b.step(5)
        b.close()
    b = abi.Batch(robots, abi.PRECISION_MIXED)
    b.choose_steps("passes")
    b.step(3 * k + 1029)
    want = resident._all(b)
    b.close()
    for g in got:
        for name in want:
            assert np.array_equal(g[name], want[name], equal_nan=True), name


def test_batches_that_keep_the_passes():
    def robot(**kw):
        return resident._body(np.random.default_rng(2), (5, 5, 5), mats=2, **kw)

    assert _plan([robot()])["many_from"] > 0
    cilia, signals = robot(enable_cilia=True), robot(enable_signals=True)
    cilia.cilia_base = np.full(cilia.grid.shape + (3,), 1e-3)
    for m in cilia.materials:
        m.cilia = 1.0
    field = robot()
    field.force_field = [("mtCONST", 1e-3), None, None]
    held = robot()
    held.bcs = [wl.BCRegion(prim=0, dof_fixed=7, x=0.0, y=0.0, z=0.0, dx=0.2, dy=1.0, dz=1.0)]
    removal = robot(secondary_experiment=True)
    removal.materials[0].remove_after = 0.001
    large = resident._body(np.random.default_rng(3), (20, 20, 20), fill=1.0)  # beyond eight thread blocks
    cases = [([robot(), r], abi.PRECISION_MIXED) for r in
             (robot(enable_collision=True), cilia, signals, field, held, robot(enable_detach=True), removal, large)]
    for robots, precision in cases + [([robot()], abi.PRECISION_FP64)]:
        b = abi.Batch(robots, precision)
        with pytest.raises(abi.Vx3gError):
            b.choose_steps("many")
        p = b.step_plan()
        assert p["many_from"] == p["launches"] == 0 and p["clusters"] == {}
        b.step(3)
        b.close()
