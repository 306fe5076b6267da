"""Undamped springs, two per packed evaluation, against the float oracle, bit for bit: rows
of even and odd length, list and per-spring stiffness, lengths inside and outside the range
of the packed square root, vertices that coincide, and positions up to and past the bound
above which every row is summed spring by spring."""
import numpy as np
import pytest

import simulator_gb300 as vs
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("perk,force_damping", [(False, 0.0), (True, 0.0), (False, -0.02)])
@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e-15, 1e-16, 1e-25, 1e8, 2.9e14, 3.1e14, 9e14, 2e15])
def test_steps_equal_the_oracle(scale, perk, force_damping):
    rng = np.random.default_rng(int(1e3 * abs(np.log10(scale))) + perk)
    n = 333
    xyz = (scale * rng.uniform(-1, 1, (n, 3))).astype(np.float32)
    xyz[rng.integers(0, n, 40)] = xyz[0]
    lists = []
    for m in (1100, 700):
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        sl = scenes._csr_from_pairs(n, a, b, xyz)
        if perk:
            sl.k = rng.uniform(0.5, 2.0, len(sl.ent)).astype(np.float32)
        lists.append(sl)
    p = reference_params(2)
    p.spring_damping, p.force_damping = 0.0, force_damping
    p.list_k[:] = (1.0, 2.0, 0.0, 0.0)
    g = vs.Simulator(xyz, lists, params=p)
    o = OracleSim(p, xyz, lists, prec=4)
    for _ in range(4):
        g.simulate(1)
        o.step(1)
        for a, b in zip(g.state()[:2], o.state()[:2]):
            assert np.array_equal(a, b.astype(np.float32), equal_nan=True)
