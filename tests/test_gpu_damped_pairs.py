"""Damped springs, two per packed evaluation with their own division, against the float
oracle, bit for bit: rows of even and odd length, list and per-spring stiffness, and
lengths and velocities inside and far outside the range of the packed square root and
division (which then take the intrinsics), mixed within a pair."""
import numpy as np
import pytest

import simulator_gb300 as vs
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("perk", [False, True])
@pytest.mark.parametrize("scale,speed", [(1.0, 0.0), (1.0, 1.0), (1.0, 1e-12), (1.0, 1e-30), (1e-16, 1e-9), (1e-25, 1.0),
                                         (1e12, 1e8), (1e-3, 1e10), (3e16, 1e-3)])
def test_steps_equal_the_oracle(scale, speed, perk):
    rng = np.random.default_rng(int(1e3 * abs(np.log10(scale))) + perk)
    n = 333
    xyz = (scale * rng.uniform(-1, 1, (n, 3))).astype(np.float32)
    lists = []
    for m in (1100, 700):
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        sl = scenes._csr_from_pairs(n, a, b, xyz)  # rows of 0 to about 10 entries, some joining a vertex to itself
        if perk:
            sl.k = rng.uniform(0.5, 2.0, len(sl.ent)).astype(np.float32)
        lists.append(sl)
    p = reference_params(2)
    p.list_k[:] = (1.0, 2.0, 0.0, 0.0)
    g = vs.Simulator(xyz, lists, params=p)
    o = OracleSim(p, xyz, lists, prec=4)
    v = rng.normal(0, 1, (n, 3)) * speed * np.exp(rng.normal(0, 4, (n, 1)))
    v[rng.random(n) < 0.2] = 0.0
    xo = (xyz.astype(np.float64) - p.dt * v).astype(np.float32)
    zero = np.zeros_like(xyz)
    g.set_state(xyz, xo, zero)
    o.set_state(xyz, xo, zero)
    for _ in range(4):
        g.simulate(1)
        o.step(1)
        for a, b in zip(g.state()[:2], o.state()[:2]):
            assert np.array_equal(a, b.astype(np.float32), equal_nan=True)
