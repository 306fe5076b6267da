"""What the adjoint holds on the device: the springs' part in x_old only where a reverse
sweep needs it (damped springs, a state out of the tame range, a replay that may leave
the forward pass's states), and gradients that do not depend on whether it is there."""
import numpy as np
import pytest

import simulator_gb300 as vs
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("damped", [False, True])
def test_bytes_held(damped):
    n = 400
    cloth = scenes.grid_cloth(n, 1.0, 0.0)
    p = scenes.physics_params(4)
    if damped:
        p.spring_damping = -1e-6
    s = vs.Simulator(cloth.xyz, cloth.lists, params=p, pinned=cloth.pinned)
    springs = sum(int(sl.row[-1]) for sl in cloth.lists)
    steps, every = 5, 2
    before = free_bytes()
    s.forward(steps, every)
    s.backward(s.positions())
    held = before - free_bytes()
    states = (steps + every - 1) // every + (every + 1) + 2  # checkpoints, a segment's record, two between
    need = springs * (136 if damped else 88) + n * n * (72 * states + 6 * 8 + 6 * 8 + 3 * 8 + 6 * 8)
    assert need <= held + (1 << 20)
    assert held <= need + 20 * (2 << 20)  # as many allocations, each rounded up to at most 2 MiB


def test_body_moved_to_where_it_was():
    cloth = scenes.grid_cloth(48, 1.0, 0.0, pin_top_corners=False)
    body = scenes.icosphere(3, 0.3, (0.0, -0.3003, 0.0))
    out = []
    for moved in (False, True):
        s = vs.Simulator(cloth.xyz, cloth.lists, body.xyz, body.tris, None, params=scenes.physics_params(4))
        s.forward(90, 20)
        assert s.forward_contacts().sum() > 0
        if moved:
            s.update_body(body.xyz, None)
        out.append(s.backward(s.positions()))
        out.append(s.backward(s.positions()))  # again, over the segment the first one replayed last
    for dk, ds in out[1:]:
        assert np.array_equal(dk, out[0][0])
        assert np.allclose(ds, out[0][1], rtol=2.0 ** -20)  # summed by atomics
