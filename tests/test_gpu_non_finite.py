"""Simulations that hold NaNs for a while, against the float oracle bit for bit: vertices
that had gone to NaN are put back and meet their body as if they had never left, and
vertices that are going to NaN meet nothing."""
import numpy as np
import pytest

import simulator_gb300 as vs
from oracle.ffi import OracleSim
from simulator_gb300 import scenes

pytestmark = pytest.mark.gpu


def scene(physics, side=64):
    cloth = scenes.grid_cloth(side, 1.0, 0.0, pin_top_corners=False)
    body = scenes.icosphere(3, 0.3, (0.0, -0.3003, 0.0))
    if physics == "workload":
        p = scenes.physics_params(4)
    else:
        p = vs.reference_params(3)
        p.gravity[1] = -0.05
        p.list_k[:] = (100.0, 60.0, 2.0, 0.0)
    return cloth, body, p


def assert_equal(gpu, oracle):
    for a, b in zip(gpu.state(), oracle.state()):
        assert np.array_equal(a, b.astype(np.float32), equal_nan=True)


@pytest.mark.parametrize("calls", [[1] * 96, [16] * 6, [1, 95]])  # single steps, graphs, both
@pytest.mark.parametrize("physics", ["workload", "reference"])
def test_vertices_put_back(physics, calls):
    cloth, body, p = scene(physics)
    g = vs.Simulator(cloth.xyz, cloth.lists, body.xyz, body.tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, body.xyz, body.tris, None, prec=4)
    everything = np.arange(len(cloth.xyz), dtype=np.uint32)
    g.update_vertices(everything, np.full_like(cloth.xyz, np.nan))
    g.simulate(3)  # both halves of the double-buffered state are NaN
    assert np.isnan(g.positions()).all()
    g.update_vertices(everything, cloth.xyz)
    for n in calls:
        g.simulate(n)
        o.step(n)
        assert_equal(g, o)
    assert g.count_contacts() > 0


@pytest.mark.parametrize("bad", [(np.nan, np.nan, np.nan), (np.nan, 0.0, 0.0), (np.inf, 0.0, 0.0)])
@pytest.mark.parametrize("physics", ["workload", "reference"])
def test_vertices_going_to_nan(physics, bad):
    cloth, body, p = scene(physics, 48)
    g = vs.Simulator(cloth.xyz, cloth.lists, body.xyz, body.tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, body.xyz, body.tris, None, prec=4)
    g.simulate(160)
    o.step(160)
    assert_equal(g, o)
    touching = np.flatnonzero(np.abs(g.state()[2]).sum(1))
    assert len(touching) > 4
    v = int(touching[len(touching) // 2])
    g.update_vertices([v], [bad])
    o.set_vertex(v, np.array(bad, np.float32))
    for _ in range(4):
        g.simulate(1)
        o.step(1)
        assert_equal(g, o)
