"""Steps whose launches overlap (one chain of fused steps) against the same steps with a
device synchronisation after each: the states are equal bit for bit, with the springs
staged or not, step by step and as graphs, with the body moved and vertices dragged in
between."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


def cloth(rows, cols):
    c, r = np.meshgrid(np.arange(cols), np.arange(rows))
    h = 1.0 / max(rows, cols)
    xyz = np.stack([(c.ravel() - cols / 2) * h, np.zeros(rows * cols), (r.ravel() - rows / 2) * h], 1).astype(np.float32)
    i = np.arange(rows * cols).reshape(rows, cols)
    a = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    b = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    return xyz, [scenes._csr_from_pairs(rows * cols, np.concatenate([a, b]), np.concatenate([b, a]), xyz)]


@pytest.mark.parametrize("physics", ["workload", "reference"])
@pytest.mark.parametrize("staged", [0, 1])
@pytest.mark.parametrize("rows,cols,margin", [(9, 33, 0), (70, 70, 0), (300, 261, 1)])
def test_equal(rows, cols, margin, staged, physics):
    xyz, lists = cloth(rows, cols)
    body = scenes.icosphere(3, 0.3, (0.0, -0.302, 0.0))
    p = scenes.physics_params(4) if physics == "workload" else reference_params(1)
    p.n_lists = 1
    p.collision_margin, p.split_collision, p.stage_neighbours = margin, 0, staged
    if physics == "reference":
        p.gravity[1] = -0.5
    one, other = [vs.Simulator(xyz, lists, body.xyz, body.tris, None, params=p) for _ in range(2)]
    for k, n in enumerate((1, 3, 16, 37, 5)):
        for s in (one, other):
            if k % 2:
                s.update_body(body.xyz + np.float32(0.01 * k) * np.array([1, 0, 0], np.float32), None)
            s.update_vertices(np.array([0], np.uint32), xyz[:1] + np.float32(1e-4 * k))
        one.simulate(n)
        for _ in range(n):
            other.simulate(1)
            other.sync()
    for a, b in zip(one.state(), other.state()):
        assert np.array_equal(a, b)
