"""Trees of more than 524,288 triangles, whose rebuild de-duplicates before it builds: few and
many equal codes (the leaves then fill more chunks than the spanning nodes stage in shared
memory, or fewer, or one chunk, or one leaf), rebuilds with few changed codes (merged) and
with most (radix passes).  Every tree equals the oracle's (integers and boxes)."""
import numpy as np
import pytest

import simulator_gb300 as vs
from helpers import lbvh_diff, soup
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


def surface(n):
    """A wavy n x n grid: many triangles share a code."""
    u = np.stack(np.meshgrid(np.linspace(-1, 1, n), np.linspace(-1, 1, n)), -1).reshape(-1, 2)
    xyz = np.stack([u[:, 0], 0.2 * np.sin(3 * u[:, 0]) * np.cos(4 * u[:, 1]), u[:, 1]], 1).astype(np.float32)
    return xyz, scenes.grid_faces(n).astype(np.uint32)


def copies(n, of):
    base, _ = soup(of, seed=of)
    v = base.reshape(-1, 3, 3)[np.random.default_rng(1).integers(0, of, n)]
    return v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


# leaves (counted by the oracle); the chunks of 448 to 512 they fill
BODIES = {
    "soup 524289": (lambda: soup(524289, seed=3, dup_frac=0.02), 513860),        # 1,148
    "soup 1100001": (lambda: soup(1100001, seed=4, dup_frac=0.3), 855312),       # 1,782
    "surface 813": (lambda: surface(813), 871740),                               # 1,703
    "copies of 400000": (lambda: copies(700000, 400000), 330372),                # 689: staged
    "copies of 300": (lambda: copies(530001, 300), 300),                         # one
    "copies of 1": (lambda: copies(530001, 1), 1),
}


@pytest.mark.parametrize("name", BODIES)
def test_equals_the_oracle(name):
    make, leaves = BODIES[name]
    xyz, tris = make()
    cloth = scenes.grid_cloth(4, 1.0, 5.0, pin_top_corners=False)
    p = reference_params(3)
    g = vs.Simulator(cloth.xyz, cloth.lists, xyz, tris, None, params=p)
    o = OracleSim(p, cloth.xyz, cloth.lists, xyz, tris, None, prec=4)
    tree = g.export_lbvh()
    assert tree["n_leaves"] == leaves
    assert lbvh_diff(tree, o.export_lbvh()) == []
    few = xyz.copy()
    few[tris[:90].ravel()] += np.float32(0.003)
    for moved in (few, few, (xyz * np.float32([0.9, 1.1, 1.0])).astype(np.float32)):
        g.update_body(moved, None)
        o.update_body(moved, None)
        assert lbvh_diff(g.export_lbvh(), o.export_lbvh()) == []
