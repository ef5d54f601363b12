"""vx3g_autotune leaves the fork point of the contact stream as the context set it unless it has timed both
(64 steps and more), and a cache entry names it only then."""

import json

import numpy as np
import pytest

from vx3g import abi
from vx3g import workloads as wl

pytestmark = pytest.mark.gpu


def _batch(cells=6):
    rng = np.random.default_rng(cells)
    m = [wl.Material(E=1e6, nu=0.35, cte=0.01)]
    return abi.Batch([wl.bernoulli_body(rng, (cells,) * 3, 0.8, m, random_phase=True, temp_vary=True, temp_amplitude=39.0,
                                        enable_collision=True) for _ in range(3)], abi.PRECISION_MIXED)


def _fork(path=None, steps=0):
    b = _batch()
    if path:
        b.autotune(steps, path)
    fork = b.step_plan()["fork"]
    b.close()
    return fork


@pytest.mark.parametrize("steps", [0, 10, 24, 40, 63, 64, 150])
def test_fork_point(tmp_path, steps):
    assert _fork() == 1  # robots that rebuild in shared memory: before the rebuild
    path = tmp_path / "cache.json"
    b = _batch()
    b.autotune(steps, path)
    fork = b.step_plan()["fork"]
    b.close()
    if steps < 24:
        assert fork == 1 and not path.exists()
        return
    entry = next(iter(json.loads(path.read_text()).values()))
    if steps < 64:
        assert fork == 1 and len(entry) == 2
    else:
        assert len(entry) == 3 and entry[2] == fork
    assert _fork(path) == fork  # as a later context reads it


@pytest.mark.parametrize("entry,fork", [([6, 6], 1), ([0, 3], 1), ([6, 6, 0], 0), ([6, 6, 1], 1)])
def test_entries(tmp_path, entry, fork):
    path = tmp_path / "cache.json"
    b = _batch()
    b.autotune(24, path)
    b.close()
    key = next(iter(json.loads(path.read_text())))
    path.write_text(json.dumps({key: entry}))
    assert _fork(path) == fork
