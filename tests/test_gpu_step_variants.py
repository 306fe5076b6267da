"""Which step kernels small garments run, from a trace of their launches: helper warps in
fused steps of one tile per CTA only, queued queries where they were asked for, and the
same states from all of them."""
import re

import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


def small_batch(split, garments=3, physics="workload"):
    if physics == "workload":
        p = scenes.physics_params(4)
    else:
        p = vs.reference_params(3)
        p.list_k[:] = (100.0, 60.0, 2.0, 0.0)
    p.split_collision = split
    p.use_graph = 0
    b = vs.BatchSimulator(p)
    for k in range(garments):
        c = scenes.grid_cloth(33 + 7 * k, 1.0, 0.0)
        body = scenes.icosphere(3, 0.3, (0.0, -0.302, 0.0))
        b.add(c.xyz, c.lists, body.xyz, body.tris, body.normals, pinned=c.pinned)
    b.finalize()
    return b


@pytest.fixture(scope="module", autouse=True)
def profiler_started():
    import torch
    for _ in range(2):  # the first trace of a process may come back empty
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]):
            torch.zeros(8, device="cuda").add_(1)
            torch.cuda.synchronize()


def step_kernels(b, steps):
    """(template arguments of every step kernel launched, collision kernels launched)"""
    import torch
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        b.step(steps)
        b.sync()
    names = [e.name for e in prof.events()]
    kernels = [re.search(r"k_step<([^>]*)>", n) for n in names]
    kernels = [[a.strip().split(")")[-1] for a in m.group(1).split(",")] for m in kernels if m]
    if not kernels:
        pytest.skip("the profiler recorded no kernels")
    return kernels, sum("k_collide" in n for n in names)


def truth(word):
    return word in ("true", "1")


@pytest.mark.parametrize("physics", ["workload", "reference"])
@pytest.mark.parametrize("garments", [1, 3])
def test_helpers_only_in_fused_steps(garments, physics):
    states = []
    for split in (1, 0):
        b = small_batch(split, garments, physics)
        b.step(40)
        kernels, collide = step_kernels(b, 4)
        helped = [truth(k[-1]) for k in kernels]
        if split and garments > 1:  # two chains, each with its queue
            assert not any(helped)
            assert collide == len(kernels)
        else:
            assert all(helped)
            assert collide == 0
        assert b.count_contacts() > 0
        states.append(b.state())
        b.close()
    for x, y in zip(*states):
        assert np.array_equal(x, y)
