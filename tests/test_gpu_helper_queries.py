"""Steps with helper warps (small simulations: queries answered beside the spring sums)
against the same steps that query every vertex every step (collision_margin off, no
helpers): the states are equal bit for bit, over sizes that leave partial warps and
tiles, both record forms, a body that stands still, turns or jumps, pins, and batches
(queued queries)."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


def cloth(rows, cols, seed):
    rng = np.random.default_rng(seed)
    c, r = np.meshgrid(np.arange(cols), np.arange(rows))
    h = 1.0 / max(rows, cols, 2)
    xyz = np.stack([(c.ravel() - cols / 2) * h, np.zeros(rows * cols), (r.ravel() - rows / 2) * h], 1)
    xyz = (xyz + rng.normal(0, 1e-3, xyz.shape)).astype(np.float32)
    i = np.arange(rows * cols).reshape(rows, cols)
    pairs = np.concatenate([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                            np.stack([i[:-1].ravel(), i[1:].ravel()], 1)])
    sl = scenes._csr_from_pairs(rows * cols, np.concatenate([pairs[:, 0], pairs[:, 1]]),
                                np.concatenate([pairs[:, 1], pairs[:, 0]]), xyz)
    return xyz, [sl]


def params(physics, margin):
    if physics == "workload":
        p = scenes.physics_params(4)
        p.n_lists = 1
    else:
        p = reference_params(1)
        p.gravity[1] = -0.5
    p.collision_margin = margin
    return p


def poses(body, motion, n):
    for k in range(n):
        if motion == "jump" and k % 3 == 2:
            yield body.xyz + np.float32(0.01) * np.array([0, (-1) ** k, 0], np.float32)
        elif motion == "turn":
            a = 0.01 * k
            r = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]])
            yield np.ascontiguousarray(body.xyz @ r, np.float32)
        else:
            yield None


@pytest.mark.parametrize("physics", ["workload", "reference"])
@pytest.mark.parametrize("rows,cols,motion", [(1, 1, "still"), (1, 31, "still"), (3, 11, "turn"), (16, 8, "jump"),
                                              (17, 19, "still"), (64, 64, "turn"), (130, 131, "jump"), (278, 280, "still")])
def test_single(rows, cols, motion, physics):
    xyz, lists = cloth(rows, cols, rows)
    body = scenes.icosphere(3, 0.3, (0.0, -0.302, 0.0))
    pins = np.array([0], np.uint32) if rows * cols > 40 else None
    sims = [vs.Simulator(xyz, lists, body.xyz, body.tris, None, params=params(physics, m), pinned=pins) for m in (1, 0)]
    contacts = 0
    for x in poses(body, motion, 12):
        for s in sims:
            if x is not None:
                s.update_body(x, None)
            s.simulate(10)
        contacts += sims[0].count_contacts()
    assert rows * cols < 4096 or contacts > 0
    for a, b in zip(sims[0].state(), sims[1].state()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("physics", ["workload", "reference"])
def test_batch(physics):
    out = []
    for m in (1, 0):
        b = vs.BatchSimulator(params(physics, m))
        for k, (r, c) in enumerate([(5, 7), (64, 33), (40, 40)]):
            xyz, lists = cloth(r, c, k)
            body = scenes.icosphere(2 + k, 0.3, (0.0, -0.302, 0.0))
            b.add(xyz, lists, body.xyz, body.tris, None, pinned=[0])
        b.finalize()
        b.step(120)
        out.append(b.state())
        assert b.count_contacts() > 0
        b.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
