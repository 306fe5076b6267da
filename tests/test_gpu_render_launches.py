"""The output stage's launches (positions and faces in one, both overlapping what is before
them) against the oracle, bit for bit: vertices with no face, one and more than the faces
whose numbers are read ahead, sizes around a block, right after steps and before more
steps."""
import numpy as np
import pytest

import simulator_gb300 as vs
from oracle import ffi
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nf", [(3, 1), (17, 40), (255, 256), (256, 257), (300, 2000), (1000, 255), (70000, 90000)])
def test_equals_the_oracle(n, nf):
    rng = np.random.default_rng(n)
    xyz = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    faces = np.stack([rng.permutation(n)[:3] if n < 300 else rng.integers(0, n, 3) for _ in range(nf)])
    faces = faces[(faces[:, 0] != faces[:, 1]) & (faces[:, 1] != faces[:, 2]) & (faces[:, 0] != faces[:, 2])]
    faces[: nf // 8, 0] = 0  # a vertex with many
    faces = np.ascontiguousarray(faces[(faces[:, 0] != faces[:, 1]) & (faces[:, 0] != faces[:, 2])], np.uint32)
    i = np.arange(n - 1)
    sl = scenes._csr_from_pairs(n, np.concatenate([i, i + 1]), np.concatenate([i + 1, i]), xyz)
    p = scenes.physics_params(4)
    p.n_lists = 1
    sim = vs.Simulator(xyz, [sl], params=p)
    sim.set_faces(faces)
    for steps in (1, 3):
        sim.simulate(steps - 1)
        before = sim.state()[0]
        sim.simulate(1)
        pos4, vn, fn = sim.render()
        want = ffi.render(sim.state()[0], before, faces)
        for a, b in zip((pos4, vn, fn), want):
            assert np.array_equal(a, b, equal_nan=True)
