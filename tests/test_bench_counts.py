"""The launch count of the benchmark line follows the way the library steps the batch."""

import bench

PASSES = dict(many_from=0, most=0, launches=0)


def test_launches_of_one_call():
    n = bench.launches_per_call
    assert n(1000, 100, PASSES, True, False, False) == 2000
    assert n(1000, 100, PASSES, False, False, False) == 2000
    many = dict(many_from=3, most=256, launches=1)
    assert n(1000, 100, many, True, False, False) == 4
    assert n(1000, 100, dict(many, launches=3), True, False, False) == 12  # one per cluster size
    assert n(2, 100, many, True, False, False) == 4  # a call of few steps goes by the passes
    assert n(256, 100, many, True, False, False) == 1 and n(257, 100, many, True, False, False) == 2
    # collisions: rebuild and evaluation, the grid's list kernel, and the displacement check
    assert n(1000, 100, PASSES, False, True, False) == 5000
    assert n(1000, 100, PASSES, True, True, False) == 4010
    assert n(1000, 100, PASSES, True, True, True) == 5010
    assert n(1050, 100, PASSES, True, True, False) == 4210
    assert n(50, 100, PASSES, True, True, False) == 201
    assert n(1000, -1, PASSES, True, True, False) == 4001  # no graphs
