"""A robot that diverges inside a launch of many steps, in every form of that kernel: alone in one CTA,
bundled with others in one CTA, in a CTA whose links take several rounds of its threads, and across a
cluster.  The step in which a link tears updates all links of the robot and moves none of its voxels
(VX3_VoxelyzeKernel.cu:252-283), whichever warp comes first, so what is left equals the passes bit for
bit, the other robots are as if they were alone, and the temperature reported is the one of that step."""

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _robot(i, dims):
    rng = np.random.default_rng(100 + i)
    mats = [wl.Material(E=float(10 ** rng.uniform(5, 7)), nu=0.35, cte=0.01) for _ in range(2)]
    return wl.bernoulli_body(rng, dims, 1.0, mats, random_phase=True, temp_vary=True, temp_amplitude=39.0, z_offset=1)


def _left(b, r):
    v, l = (slice(int(o[r]), int(o[r + 1])) for o in (b.voxel_offset, b.link_offset))
    out = {k: a[v] for k, a in dict(b.state(), **{k: x for k, x in b.voxel_aux().items() if k != "contact"}).items()}
    out.update({k: a[l] for k, a in b.links().items()})
    return dict(out, time=b.time()[r], status=b.status()[r])


def _tear(b, r):
    """Sets the positions back (as a sum of two floats, a tie may be split the other way); in robot r, if
    given, with one voxel far away, so that its links' strain passes 100."""
    pos = b.state()["pos"]
    if r is not None:
        pos[b.voxel_offset[r + 1] - 1] += 50.0
    b.set_state(pos=pos)


# (robots, cells): 64 voxels in one CTA; several robots in one CTA; 636 links for the 384 threads of a
# CTA that shares its SM; a cluster of two; a cluster of eight
FORMS = [(1, (4, 4, 4)), (40, (2, 2, 3)), (300, (6, 6, 7)), (3, (6, 6, 5)), (2, (11, 11, 11))]


@pytest.mark.parametrize("count,dims", FORMS)
@pytest.mark.parametrize("steps", [1, 2, 37])
def test_a_torn_robot(count, dims, steps):
    robots = [_robot(i, dims) for i in range(count)]
    torn = count // 2
    others = sorted({0, count - 1} - {torn})

    def run(which, passes, tear):
        b = abi.Batch([robots[r] for r in which], abi.PRECISION_MIXED)
        b.choose_steps("passes" if passes else "many")
        b.step(10)
        _tear(b, which.index(torn) if tear else None)
        b.step(steps)
        out = {r: _left(b, which.index(r)) for r in {torn, *others} & set(which)}
        b.close()
        return out

    want = run([torn], True, True)[torn]
    b = abi.Batch([robots[torn]], abi.PRECISION_MIXED)
    b.step(11)
    want["tempe"] = b.voxel_aux()["tempe"]  # of the step that diverged
    b.close()
    for _ in range(4):
        got = run(list(range(count)), False, True)
        assert got[torn]["status"] == 1 and want["status"] == 1
        for k in want:
            assert np.array_equal(got[torn][k], want[k], equal_nan=True), k
        for r in others:
            alone = run([r], True, False)[r]
            for k in alone:
                assert np.array_equal(got[r][k], alone[k], equal_nan=True), (r, k)
