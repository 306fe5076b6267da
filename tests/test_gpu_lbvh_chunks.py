"""Trees whose build takes chunks of other lengths than a CTA's threads: sizes at which the
length changes (one round of chunks of 256, of more, a second and third round, and where
the summaries stop fitting shared memory), with runs of equal codes.  Every tree equals the
oracle's (integers and boxes)."""
import numpy as np
import pytest

import simulator_gb300 as vs
from helpers import lbvh_diff, soup
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 513, 77824, 77825, 97281, 155648, 155649, 311297, 466945, 524288, 524289])
def test_equals_the_oracle(n):
    xyz, tris = soup(n, seed=n, dup_frac=0.05)
    cloth = scenes.grid_cloth(4, 1.0, 5.0, pin_top_corners=False)
    p = reference_params(3)
    g = vs.Simulator(cloth.xyz, cloth.lists, xyz, tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, xyz, tris, None, prec=4)
    assert lbvh_diff(g.export_lbvh(), o.export_lbvh()) == []
    moved = np.ascontiguousarray(xyz + np.float32(0.01), np.float32)
    g.update_body(moved, None)
    o.update_body(moved, None)
    assert lbvh_diff(g.export_lbvh(), o.export_lbvh()) == []
