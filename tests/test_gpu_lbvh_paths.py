"""The rebuild's sorts and the chunk build where they change hands: bodies whose codes
nearly all change (buckets cut by the last order), that leave one bucket overfull (the
radix passes), sizes around a chunk, a bucket and the limits of each path, and runs of
equal codes that cross chunks.  Every tree equals the oracle's (integers and boxes)."""
import numpy as np
import pytest

import simulator_gb300 as vs
from helpers import lbvh_diff, soup
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu


def pair(xyz, tris, normals=None):
    cloth = scenes.grid_cloth(4, 1.0, 5.0, pin_top_corners=False)
    p = reference_params(3)
    return (vs.Simulator(cloth.xyz, cloth.lists, xyz, tris, normals, params=p),
            OracleSim(p, cloth.xyz, cloth.lists, xyz, tris, normals, prec=4))


def rebuild(g, o, xyz, normals=None):
    xyz = np.ascontiguousarray(xyz, np.float32)
    g.update_body(xyz, normals)
    o.update_body(xyz, normals)
    a = g.export_lbvh()
    assert lbvh_diff(a, o.export_lbvh()) == []
    return a


@pytest.mark.parametrize("n", [1, 2, 31, 511, 512, 513, 1024, 1025, 2047, 2049, 19584, 32768, 32769, 65537])
def test_turning_soups(n):
    """Every code changes at every rebuild."""
    xyz, tris = soup(n, seed=n, dup_frac=0.1)
    g, o = pair(xyz, tris)
    assert lbvh_diff(g.export_lbvh(), o.export_lbvh()) == []
    for a in (0.3, 0.9):
        c, s = np.cos(a), np.sin(a)
        rebuild(g, o, xyz @ np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]]))


@pytest.mark.parametrize("name", ["capsules", "ico6"])
def test_turning_bodies_with_normals(name):
    b = scenes.three_capsules() if name == "capsules" else scenes.icosphere(6, 0.4)
    g, o = pair(b.xyz, b.tris, b.normals)
    for k in range(4):
        c, s = np.cos(0.05 * k), np.sin(0.05 * k)
        r = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]])
        rebuild(g, o, (1.0 + 0.02 * k) * (b.xyz @ r), np.ascontiguousarray(b.normals @ r, np.float32))


@pytest.mark.parametrize("n", [6000, 40000])
def test_overfull_bucket_falls_back(n):
    """The last order spreads over the whole box; now all but a few triangles crowd into
    one corner, below the first splitter: that bucket overflows and the radix passes
    sort.  Then back, from the order they left."""
    xyz, tris = soup(n, seed=5)
    g, o = pair(xyz, tris)
    crowd = xyz.reshape(-1, 3, 3).copy()
    crowd[50:] = crowd[50:] * 0.004 - 0.99
    rebuild(g, o, crowd.reshape(-1, 3))
    rebuild(g, o, xyz)


@pytest.mark.parametrize("copies", [2, 33, 200, 700, 1500])
def test_runs_of_equal_codes_across_chunks(copies):
    """Each triangle `copies` times: runs longer than a warp, a chunk and a bucket."""
    base, _ = soup(max(1, 6000 // copies), seed=copies)
    v = np.repeat(base.reshape(-1, 3, 3), copies, axis=0)
    rng = np.random.default_rng(2)
    v = v[rng.permutation(len(v))]
    tris = np.arange(3 * len(v), dtype=np.uint32).reshape(-1, 3)
    g, o = pair(v.reshape(-1, 3), tris)
    assert lbvh_diff(g.export_lbvh(), o.export_lbvh()) == []
    a = rebuild(g, o, (v[:, :, [2, 0, 1]]).reshape(-1, 3))
    assert a["n_leaves"] <= len(base) // 3
    rebuild(g, o, v.reshape(-1, 3) + np.float32(1e-5))
