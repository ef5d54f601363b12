"""Every compiled launch shape of the two mixed-precision passes leaves the same bits, also with contacts,
cilia, a force field, boundary conditions, detaching links and robots that stop: the shapes differ in when a
thread loads its links' and materials' data, not in what it computes.  Voxel counts around a block of 64 and
128 threads and a warp."""

import json

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu

SHAPES = 8


def _robots():
    out = []
    for i, dims in enumerate([(1, 1, 1), (31, 1, 1), (4, 4, 4), (13, 5, 1), (8, 4, 4), (9, 7, 6)]):
        rng = np.random.default_rng(i)
        mats = [wl.Material(E=float(10 ** rng.uniform(5, 6)), nu=0.35, cte=0.01, cilia=0.5),
                wl.Material(E=2e5, nu=0.0, cte=0.01, thermal_on_after=0.001 * (i % 2), fail_stress=4e3 if i == 5 else 0.0)]
        r = wl.bernoulli_body(rng, dims, 1.0, mats, random_phase=True, temp_vary=True, temp_amplitude=39.0,
                              enable_collision=i != 2, enable_expansion=1, z_offset=i % 2, slow_damping=0.01 * (i % 3))
        if i == 3:
            r.enable_cilia = True
            r.cilia_base = 1e-2 * rng.standard_normal(r.grid.shape + (3,))
        if i == 4:
            r.bcs = [wl.BCRegion(prim=0, dof_fixed=7, x=0.0, y=0.0, z=0.0, dx=0.2, dy=1.0, dz=1.0)]
            r.force_field = [("mtCONST", 1e-3), None, None]
        r.enable_detach = i == 5
        out.append(r)
    return out


def _run(path=None):
    b = abi.Batch(_robots(), abi.PRECISION_MIXED)
    if path:
        b.autotune(0, path)
    b.step(60)
    b.stop_robot(1)
    b.step(130)
    out = dict(b.state(), **b.links(), **b.voxel_aux())
    b.close()
    return out


def test_all_shapes(tmp_path):
    probe = tmp_path / "probe.json"
    b = abi.Batch(_robots(), abi.PRECISION_MIXED)
    b.autotune(64, probe)
    b.close()
    key = next(iter(json.loads(probe.read_text())))
    want = _run()
    assert np.abs(want["contact"]).max() > 0
    for k in range(SHAPES):
        path = tmp_path / f"{k}.json"
        path.write_text(json.dumps({key: [k, (k + 3) % SHAPES, 0]}))
        got = _run(path)
        for name in want:
            assert np.array_equal(got[name], want[name], equal_nan=True), (k, name)


@pytest.mark.parametrize("cells,threads", [(2, 32), (10, 32), (40, 64), (60, 256)])
def test_fp64_shapes_follow_the_batch(cells, threads):
    """Blocks of one warp until each of the 152 SMs has eight: 38,912 voxels, then wider ones."""
    b = abi.Batch([wl.solid_block(cells)], abi.PRECISION_FP64)
    assert list(b.launch_shapes())[2:] == [threads, 1]
    b.close()
