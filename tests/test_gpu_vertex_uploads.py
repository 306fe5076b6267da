"""Vertex updates that the kernel reads from the staging buffer: calls one after another
without a wait (the buffer is reused and grows), sizes around a block, steps before and
after, against the same calls with a synchronisation after each; the states are equal bit
for bit, and the moved vertices are where they were put."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, 1, 17])
@pytest.mark.parametrize("side", [16, 128])
def test_equal(side, steps):
    cloth = scenes.grid_cloth(side, 1.0, 0.0)
    body = scenes.icosphere(3, 0.3, (0.0, -0.302, 0.0))
    n = side * side
    sims = [vs.Simulator(cloth.xyz, cloth.lists, body.xyz, body.tris, body.normals, params=scenes.physics_params(4),
                         pinned=cloth.pinned) for _ in range(2)]
    rng = np.random.default_rng(side)
    for m in (1, 9, 255, 256, 1, 200, min(n, 2000), 3, n):
        idx = rng.permutation(n)[:m].astype(np.uint32)
        xyz = (cloth.xyz[idx] + rng.normal(0, 1e-4, (m, 3))).astype(np.float32)
        for k, s in enumerate(sims):
            s.update_vertices(idx, xyz)
            if k:
                s.sync()
            s.simulate(steps)
            if k:
                s.sync()
        if steps == 0:
            assert np.array_equal(sims[0].positions()[idx], xyz)
    for a, b in zip(sims[0].state(), sims[1].state()):
        assert np.array_equal(a, b)
