"""The adjoint's kernels at the shapes where their tiling can go wrong: rows longer than
a chunk of springs, vertices without springs, vertex counts around a tile, segments with
a remainder, the recorded last segment, and a trajectory that leaves the range in which
the zero damping term is left out."""
import numpy as np
import pytest

import simulator_gb300 as vs
from oracle.ffi import OracleSim
from simulator_gb300 import scenes
from simulator_gb300.params import reference_params

pytestmark = pytest.mark.gpu

# both sides work in FP64 and return floats: a float rounding (2^-24 of the value, at most of the
# largest gradient), with a factor 16 for the FP64 rounding that some hundred steps carry along
TOL = 2.0 ** -20


def star(n: int, hub: int, seed: int):
    """Vertex 0 joined to 1..hub in list 0, a chain over the first two thirds of the rest
    in list 1, the others without springs; random positions, rest lengths 2 % short."""
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32)
    pairs0 = [(0, k) for k in range(1, min(hub, n - 1) + 1)]
    end = hub + 1 + 2 * (n - hub - 1) // 3
    pairs1 = [(k, k + 1) for k in range(hub + 1, end - 1)]
    lists = []
    for pairs in (pairs0, pairs1):
        a = np.array(pairs, np.int64).reshape(-1, 2)
        sl = scenes._csr_from_pairs(n, np.concatenate([a[:, 0], a[:, 1]]), np.concatenate([a[:, 1], a[:, 0]]), xyz)
        sl.ent["rest"] *= np.float32(0.98)
        lists.append(sl)
    return xyz, lists


def params(damped: bool, force_damping: float = 0.0):
    p = reference_params(2)
    p.list_k[:] = (2.0, 5.0, 0.0, 0.0)
    if not damped:
        p.spring_damping, p.verlet_damping, p.force_damping = 0.0, 0.97, force_damping
    return p


def check(xyz, lists, p, steps, every, pinned=None):
    g = vs.Simulator(xyz, lists, params=p, pinned=pinned)
    o = OracleSim(p, xyz, lists, prec=8, pinned=pinned)
    g.forward(steps, every)
    o.forward(steps, every)
    x = g.positions()
    assert np.array_equal(x, o.state()[0].astype(np.float32))
    dl = (x + np.float32(0.01) * np.sin(np.arange(x.size, dtype=np.float32)).reshape(x.shape)).astype(np.float32)
    dk, ds = g.backward(dl)
    odk, ods = o.backward(dl.astype(np.float64))
    assert np.abs(dk - odk).max() <= TOL * np.abs(odk).max()
    assert np.abs(ds - ods).max() <= TOL * np.abs(ods).max()
    return g, dl, dk, ds


@pytest.mark.parametrize("damped", [False, True])
@pytest.mark.parametrize("n,hub", [(2, 1), (33, 8), (152 * 32 + 1, 5), (900, 384), (1300, 800)])
def test_rows_and_tiles(n, hub, damped):
    xyz, lists = star(n, hub, n)
    check(xyz, lists, params(damped), 12, 5, pinned=np.array([n - 1], np.uint32))


@pytest.mark.parametrize("steps,every", [(1, 1), (7, 3), (6, 3), (4, 9), (5, 1)])
def test_segments_and_a_second_backward(steps, every):
    xyz, lists = star(300, 40, 5)
    g, dl, dk, _ = check(xyz, lists, params(False, -0.01), steps, every)
    dk2, _ = g.backward(dl)  # the record now holds the first segment: all others are replayed
    assert np.array_equal(dk, dk2)
    g.set_pinned(np.array([0, 7], np.uint32))  # a backward pass takes the pins as they are
    if every >= steps:
        b = vs.Simulator(xyz, lists, params=params(False, -0.01), pinned=np.array([0, 7], np.uint32))
        b.forward(steps, every)
        assert np.array_equal(g.backward(dl)[0], b.backward(dl)[0])


def test_beyond_the_range_of_the_left_out_term():
    """An unstable step size takes positions past 1e100 (and not to infinity)."""
    xyz, lists = star(200, 60, 9)
    p = params(False)
    p.list_k[:] = (2.0e6, 5.0e6, 0.0, 0.0)
    g = vs.Simulator(xyz, lists, params=p)
    o = OracleSim(p, xyz, lists, prec=8)
    g.forward(26, 8)
    o.forward(26, 8)
    with np.errstate(over="ignore", invalid="ignore"):
        ox = o.state()[0]
        assert np.abs(ox).max() > 1e100 and np.isfinite(ox).all()
        assert np.array_equal(g.positions(), ox.astype(np.float32))
