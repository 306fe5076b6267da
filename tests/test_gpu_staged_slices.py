"""Steps whose warps stage their slices' springs in shared memory against steps that read
them from global memory: the states are equal bit for bit, over garments with partial
slices, rows too long for the stage buffers, slices without springs and single vertices,
in one chain and two, for every CTA size and several grids."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


def batch(physics, staged, split, chains, perk):
    p = scenes.physics_params(4) if physics == "workload" else reference_params(1)
    p.n_lists = 1
    p.stage_neighbours, p.split_collision, p.overlap_groups = staged, split, chains
    b = vs.BatchSimulator(p)
    for k, (n, per) in enumerate([(1, 0), (31, 3), (33, 2.5), (1000, 8), (257, 40), (64, 0), (1025, 5), (96, 11)]):
        rng = np.random.default_rng(k)
        xyz = rng.uniform(-0.3, 0.3, (n, 3)).astype(np.float32)
        xyz[:, 1] = 0.05 * rng.random(n)
        m = int(n * per / 2)
        i, j = rng.integers(0, n, m), rng.integers(0, n, m)
        if k == 3:  # its last slices have no springs
            i, j = i % 800, j % 800
        sl = scenes._csr_from_pairs(n, np.concatenate([i, j]), np.concatenate([j, i]), xyz)
        if perk:
            sl.k = rng.uniform(0.5, 2.0, len(sl.ent)).astype(np.float32)
        body = scenes.icosphere(2, 0.3, (0.0, -0.302, 0.0))
        b.add(xyz, [sl], body.xyz, body.tris, None, pinned=[0])
    b.finalize()
    return b


@pytest.mark.parametrize("physics,split,chains,perk", [("workload", 0, 0, False), ("workload", 1, 0, False),
                                                       ("workload", 0, 1, True), ("reference", 0, 0, False),
                                                       ("reference", 1, 1, True)])
def test_equal(physics, split, chains, perk):
    plain = batch(physics, 0, split, chains, perk)
    plain.step(37)
    want = plain.state()
    for blk, ctas in [(128, 0), (128, 1), (128, 2), (256, 1), (512, 0), (1024, 1)]:
        b = batch(physics, 1, split, chains, perk)
        b.set_launch(blk, ctas)
        assert b.launch_info()["stage_neighbours"] == 1
        b.step(37)
        for x, y in zip(b.state(), want):
            assert np.array_equal(x, y, equal_nan=True)
        b.close()
