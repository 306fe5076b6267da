"""Simulations that hold NaNs, against the float oracle bit for bit: vertices that had gone
to NaN are put back and meet their body as if they had never left, vertices that are going
to NaN meet nothing, and triangles whose corners are NaN are met by nothing."""
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


def broken_body(seed, inf=False, partly=False):
    """A sphere of separate triangles; of 40 % of them all corners are NaN on one axis or on
    all (with `inf`, infinite instead), with `partly` also a single one."""
    b = scenes.icosphere(4, 0.3, (0.0, -0.3003, 0.0))
    rng = np.random.default_rng(seed)
    v = b.xyz[b.tris].copy()
    for t in np.flatnonzero(rng.random(len(v)) < 0.4):
        bad = rng.choice([np.inf, -np.inf]) if inf else np.nan
        axes = slice(None) if rng.random() < 0.3 else rng.integers(3)
        if not partly or rng.random() < 0.8:
            v[t, :, axes] = bad
        else:
            v[t, rng.integers(3), axes] = bad
    return v.reshape(-1, 3), np.arange(3 * len(v), dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("inf", [False, True])
def test_queries_of_a_broken_body(inf):
    cloth, _, p = scene("workload", 8)
    xyz, tris = broken_body(1, inf, True)
    g = vs.Simulator(cloth.xyz, cloth.lists, xyz, tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, xyz, tris, None, prec=4)
    tree, ref = g.export_lbvh(), o.export_lbvh()
    for k in tree:
        assert np.array_equal(tree[k], ref[k], equal_nan=True), k
    rng = np.random.default_rng(2)
    d = rng.normal(0, 1, (40000, 3))
    pts = (d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.28, 0.31, (len(d), 1)) + [0, -0.3003, 0])
    pts = pts.astype(np.float32)
    pts[:300, rng.integers(0, 3, 300)] = np.inf
    pts[300:600] *= np.where(rng.random((300, 3)) < 0.5, np.inf, 1.0).astype(np.float32)
    pts[600:700, 1] = np.nan
    a, b = g.query(pts), o.query(pts)
    assert (a[0] >= 0).sum() > (0 if inf else 4000)  # an infinite body has few distinct codes
    for x, y in zip(a, b):
        assert np.array_equal(x, np.asarray(y, x.dtype), equal_nan=x.dtype.kind == "f")


@pytest.mark.parametrize("margin", [1, 0])
@pytest.mark.parametrize("physics", ["workload", "reference"])
def test_steps_onto_a_broken_body(physics, margin):
    cloth, body, p = scene(physics)
    p.collision_margin = margin
    xyz, tris = broken_body(3)
    b = scenes.icosphere(4, 0.3, (0.0, -0.3003, 0.0))
    whole = b.xyz[b.tris].reshape(-1, 3)
    g = vs.Simulator(cloth.xyz, cloth.lists, whole, tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, whole, tris, None, prec=4)
    for s in (g, o):
        s.update_body(xyz, None)
    for n in [1] * 8 + [16] * 9:
        g.simulate(n)
        o.step(n)
        assert_equal(g, o)
    assert g.count_contacts() > 0
    assert not np.isnan(g.positions()).any()
