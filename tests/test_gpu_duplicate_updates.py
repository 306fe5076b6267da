"""update_vertices with vertices named several times: the last position wins, whether the
duplicates share a warp of the update's kernel, lie blocks apart, or come in many calls
(more than the marks that find them count to), for single simulators and batches."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


def last_wins(x, idx, xyz):
    x = x.copy()
    for i, p in zip(idx, xyz):
        x[i] = p
    return x


@pytest.mark.parametrize("batch", [False, True])
def test_last_wins(batch):
    cloth = scenes.grid_cloth(64, 1.0, 0.0)
    if batch:
        s = vs.BatchSimulator(scenes.physics_params(4))
        s.add(cloth.xyz, cloth.lists)
        s.add(cloth.xyz, cloth.lists)
        s.finalize()
    else:
        s = vs.Simulator(cloth.xyz, cloth.lists, params=scenes.physics_params(4))
    x = s.positions()
    n = len(x)
    rng = np.random.default_rng(0)
    cases = [np.array([5, 5]), np.repeat([7, 3, 9], 11), np.zeros(1000, int), rng.integers(0, n, 3000),
             rng.integers(0, 40, 5000), np.concatenate([np.arange(n), np.arange(n)]), np.arange(n)[::-1],
             np.concatenate([np.arange(2000), [0]])]
    cases += [rng.integers(0, 16, 33) for _ in range(300)]
    for idx in cases:
        xyz = rng.normal(0, 1, (len(idx), 3)).astype(np.float32)
        s.update_vertices(idx, xyz)
        x = last_wins(x, idx, xyz)
        assert np.array_equal(s.positions(), x)
