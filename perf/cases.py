"""The work that users of the cloth simulator have it do, as measurable cases.

Each case is one pass of a program that keeps a simulator and calls it again and
again: a frame of an interactive scene, a run of steps, a frame of an animated body, a
step of a garment batch, an iteration of a stiffness fit, a body tree for a caller with
its own allocator, the output arrays of a frame.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what the program has in hand before the call
    run(state)            one pass; its outputs
    work(case)            bytes and operations one pass cannot do without
    exact(case, seed)     the outputs in 64 bits, by plain numpy and torch

Kinds of cases ("do"):
    drag      targets for a few dragged vertices, steps, positions on the device
    steps     simulate(n), positions on the device
    body      new body vertices (device arrays), steps, positions; `frames` of them
    batch     steps of many garments, positions on the device
    stream    per frame: targets of the pinned vertices from host memory, a step of many
              garments, all positions read back to page-locked memory, three in flight
    fit       state reset, forward, loss gradient on the host, backward
    tree      the body tree built into the caller's device arrays
    output    steps, then vec4 positions, vertex and face normals on the device

Two sets of physics are in use: "workload" (the stiff sheets of the benchmark, 4 steps
per 1 ms frame, no spring damping) and "reference" (the reference program's constants,
with spring and force damping).
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import simulator_gb300 as vs
from simulator_gb300 import scenes


def listed():
    return [
        # The smallest call: one step per displayed frame while the user drags a corner
        # of a 64 x 64 sheet (the smallest configured one), reference constants, as created.
        dict(name="drag_small", do="drag", rows=64, cols=64, physics="reference", body="ico4", gap=0.2, steps=1,
             settle=0, tune=False),
        # The smallest configured workload run at length: 50 frames of 4 steps in one call.
        dict(name="run_small", do="steps", rows=64, cols=64, physics="workload", body="ico4", gap=0.2, steps=200,
             settle=0, tune=True),
        # A garment mesh of the demo's size (about 16.7 K vertices, springs from its
        # triangles, odd sides) lying on its body, reference constants, as created.
        dict(name="run_garment", do="steps", rows=131, cols=127, physics="reference", body="capsules", gap=0.01,
             steps=20, settle=240, tune=False),
        # Garment-scale sheet over a body that translates: new vertices before every step.
        dict(name="body_slide", do="body", rows=112, cols=112, physics="workload", body="capsules", motion="slide",
             gap=0.1, frames=4, steps=1, settle=1600, tune=True),
        # The same body animated: it turns and breathes, one new pose per frame of 4 steps,
        # so that most of its triangles change their place in the tree's order.
        dict(name="body_turn", do="body", rows=112, cols=112, physics="workload", body="capsules", motion="turn",
             gap=0.1, frames=2, steps=4, settle=1600, tune=True),
        # The large sheet over the large oscillating body, new vertices before every step.
        dict(name="body_large", do="body", rows=512, cols=512, physics="workload", body="ico7", motion="slide",
             gap=0.2, frames=4, steps=1, settle=1600, tune=True),
        # Many draped garments of uneven size (32 to 256 vertices a side), each on its own sphere.
        dict(name="batch_draped", do="batch", garments=44, lo=32, hi=256, physics="workload", steps=16, settle=2400,
             tune=True),
        # The same, driven from host memory and read back every step.
        dict(name="batch_stream", do="stream", garments=24, lo=32, hi=160, physics="workload", frames=6, settle=1600,
             tune=True),
        # An iteration of a stiffness fit on the 128 x 128 sheet: 100 steps, a checkpoint every 25.
        dict(name="fit_sheet", do="fit", rows=128, cols=128, physics="workload", body="ico4", gap=0.2, steps=100,
             every=25),
        # The same on a small garment mesh with the reference constants (damped springs).
        dict(name="fit_garment", do="fit", rows=57, cols=43, physics="reference", body="ico3", gap=0.2, steps=60,
             every=20),
        # A body tree of 19,584 triangles for a caller with its own allocator; 3 poses.
        dict(name="tree", do="tree", body="capsules", poses=3),
        # A frame of the large sheet for a renderer: 4 steps, positions and normals.
        dict(name="output_large", do="output", rows=512, cols=512, physics="workload", body="ico5", gap=0.2, steps=4,
             settle=0, tune=True),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def sheet(lo, hi):
        rows = log_int(lo, hi)
        if rng.random() < 0.5:
            return dict(rows=rows, cols=rows, physics=rng.choice(["workload", "reference"]))
        return dict(rows=rows, cols=max(8, min(hi, int(rows * rng.uniform(0.6, 1.6)))), physics="reference")

    do = rng.choice(["drag", "steps", "steps", "body", "body", "batch", "batch", "stream", "fit", "fit", "tree", "output"])
    if do == "drag":
        return dict(do=do, **sheet(24, 256), body=rng.choice(["ico2", "ico3", "ico4"]), gap=0.2, steps=rng.randint(1, 4),
                    settle=rng.choice([0, 300]), tune=rng.random() < 0.5)
    if do == "steps":
        return dict(do=do, **sheet(24, 420), body=rng.choice(["ico3", "ico4", "ico5", "capsules"]), gap=0.02,
                    steps=log_int(3, 150), settle=rng.choice([0, 400]), tune=rng.random() < 0.5)
    if do == "body":
        return dict(do=do, **sheet(32, 420), body=rng.choice(["ico2", "ico3", "ico5", "ico6", "capsules"]),
                    motion=rng.choice(["slide", "turn"]), gap=0.05, frames=rng.randint(1, 4), steps=rng.randint(1, 4),
                    settle=400, tune=rng.random() < 0.5)
    if do == "batch":
        lo = log_int(12, 64)
        return dict(do=do, garments=log_int(2, 44), lo=lo, hi=rng.randint(lo + 8, 200),
                    physics=rng.choice(["workload", "workload", "reference"]), steps=rng.randint(1, 16),
                    settle=rng.choice([0, 1200]), tune=rng.random() < 0.5)
    if do == "stream":
        lo = log_int(12, 48)
        return dict(do=do, garments=log_int(2, 24), lo=lo, hi=rng.randint(lo + 8, 150), physics="workload",
                    frames=rng.randint(1, 6), settle=rng.choice([0, 600]), tune=rng.random() < 0.5)
    if do == "fit":
        steps = log_int(8, 100)
        return dict(do=do, **sheet(16, 120), body=rng.choice(["ico2", "ico4"]), gap=0.2, steps=steps,
                    every=rng.randint(max(1, steps // 6), steps))
    if do == "tree":
        return dict(do=do, body=rng.choice(["ico0", "ico1", "ico2", "ico3", "ico4", "ico5", "soup"]),
                    poses=rng.randint(1, 6))
    return dict(do=do, **sheet(24, 512), body=rng.choice(["ico2", "ico4"]), gap=0.2, steps=rng.randint(1, 4), settle=0,
                tune=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=256)
def _sheet(rows: int, cols: int):
    """(flat positions, faces, spring lists): a square sheet has the workloads' three
    spring families, any other sheet is a triangle mesh with its two lists."""
    if rows == cols:
        c = scenes.grid_cloth(rows, 1.0, 0.0)
        return c.xyz, c.faces, c.lists
    h = 1.0 / (max(rows, cols) - 1)
    c, r = np.meshgrid(np.arange(cols), np.arange(rows))
    xyz = np.stack([(c.ravel() - (cols - 1) / 2) * h, np.zeros(rows * cols), (r.ravel() - (rows - 1) / 2) * h], 1)
    idx = np.arange(rows * cols).reshape(rows, cols)
    a, b, d, e = idx[:-1, :-1].ravel(), idx[:-1, 1:].ravel(), idx[1:, :-1].ravel(), idx[1:, 1:].ravel()
    faces = np.concatenate([np.stack([a, d, b], 1), np.stack([b, d, e], 1)]).astype(np.uint32)
    xyz = np.ascontiguousarray(xyz, np.float32)
    return xyz, faces, vs.springs_from_mesh(xyz, faces)


@functools.lru_cache(maxsize=16)
def _body(name: str):
    """A unit body: icosphere of radius 0.3, the torso with two arms, or a triangle soup."""
    if name == "capsules":
        return scenes.three_capsules((0.0, 0.0, 0.0))
    if name == "soup":
        g = np.random.default_rng(3)
        n = 9000
        c = g.uniform(-0.4, 0.4, (n, 1, 3))
        xyz = (c + g.normal(0, 0.01, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
        nrm = g.normal(0, 1, xyz.shape)
        nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
        return scenes.Body(xyz, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), nrm.astype(np.float32))
    s = int(name[3:])
    return scenes.icosphere(s, 0.3, noise=0.02 if s == 7 else 0.0, seed=0)


def _params(case):
    if case["physics"] == "workload":
        return scenes.physics_params(4)
    return vs.reference_params(3 if case["rows"] == case["cols"] else 2)


def _pins(rows, cols):
    return np.array([0, cols - 1], np.uint32)


def _cloth_positions(case, g):
    """The flat sheet with the configured jitter (1e-4 m)."""
    xyz, _, _ = _sheet(case["rows"], case["cols"])
    return (xyz + g.normal(0.0, 1e-4, xyz.shape)).astype(np.float32)


def _body_positions(case):
    b = _body(case["body"])
    return (b.xyz - np.array([0.0, float(b.xyz[:, 1].max()) + case["gap"], 0.0])).astype(np.float32)


def _stiffness(case, lists, p, g):
    """Per-entry stiffness k exp(N(0, 0.2)), equal both ways of a spring."""
    out = []
    for l, sl in enumerate(lists):
        src = np.repeat(np.arange(len(sl.row) - 1), np.diff(sl.row.astype(np.int64)))
        end = sl.ent["end"].astype(np.int64)
        key = np.minimum(src, end) * len(sl.row) + np.maximum(src, end)
        uniq, inv = np.unique(key, return_inverse=True)
        out.append((p.list_k[l] * np.exp(g.normal(0.0, 0.2, len(uniq))))[inv].astype(np.float32))
    return out


def _poses(case, base, normals, count, g):
    """`count` device poses of a moving body, there and back again, with their normals."""
    t = np.minimum(np.arange(count), count - np.arange(count)) / 8.0 + g.uniform(0, 1)
    b = torch.from_numpy(base).cuda().double()
    n = torch.from_numpy(normals).cuda().double()
    c = b.mean(0)
    pos, nrm = [], []
    for k in range(count):
        if case.get("motion", "turn") == "slide":  # 0.5 m/s at 0.25 ms a step
            pos.append((b - torch.tensor([0.0, 0.001 * t[k], 0.0], device="cuda", dtype=torch.float64)).float())
            nrm.append(n.float())
        else:  # about 1 rad/s at 1 ms a frame, and a breath of 1 %
            a = 0.008 * t[k]
            r = torch.tensor([[math.cos(a), 0.0, math.sin(a)], [0.0, 1.0, 0.0], [-math.sin(a), 0.0, math.cos(a)]],
                             device="cuda", dtype=torch.float64)
            s = 1.0 + 0.01 * math.sin(0.3 * t[k])
            pos.append((c + s * ((b - c) @ r.T)).float())
            nrm.append((n @ r.T).float())
    return torch.stack(pos).contiguous(), torch.stack(nrm).contiguous()


def _ptr(t):
    return None if t is None else t.data_ptr()


# ---------------------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------------------
def _single(case, seed):
    g = np.random.default_rng(seed)
    _, faces, lists = _sheet(case["rows"], case["cols"])
    p = _params(case)
    x0 = _cloth_positions(case, g)
    body, bx = _body(case["body"]), _body_positions(case)
    sim = vs.Simulator(x0, lists, bx, body.tris, body.normals, params=p, pinned=_pins(case["rows"], case["cols"]))
    if case.get("settle"):
        sim.simulate(case["settle"])
    if case.get("tune"):
        sim.autotune()
    return g, sim, p, x0, bx, body, faces


def _targets(x0, rows, cols, g):
    """Where the user drags one corner block of the sheet, frame by frame (8 frames)."""
    idx = (np.arange(3)[:, None] * cols + np.arange(min(3, cols))[None, :]).ravel().astype(np.uint32) + np.uint32(
        cols * (rows // 2))
    step = g.normal(0.0, 2e-4, (8, 1, 3)).cumsum(0)
    return idx, (x0[idx][None] + step).astype(np.float32)


def prepare(case, seed):
    do = case["do"]
    s = dict(case=case, do=do, k=0)
    if do in ("batch", "stream"):
        g = np.random.default_rng(seed)
        sides = np.random.default_rng(7).integers(case["lo"], case["hi"] + 1, case["garments"])
        subs = np.random.default_rng(8).integers(3, 7, case["garments"])
        p = scenes.physics_params(4) if case["physics"] == "workload" else vs.reference_params(3)
        b = vs.BatchSimulator(p)
        pins, off, pos = [], 0, []
        for n, sub in zip(sides, subs):
            n = int(n)
            xyz, _, lists = _sheet(n, n)
            body = _body(f"ico{sub}")
            r = g.uniform(0.2, 0.4)
            x = (xyz + g.normal(0.0, 1e-4, xyz.shape)).astype(np.float32)
            bx = (body.xyz * (r / 0.3) + np.array([0.0, -0.5, 0.0])).astype(np.float32)
            b.add(x, lists, bx, body.tris, body.normals, pinned=_pins(n, n))
            pins.append(off + _pins(n, n))
            pos.append(x[_pins(n, n)])
            off += n * n
        b.finalize()
        if case["settle"]:
            b.step(case["settle"])
        if case["tune"]:
            b.autotune()
        s.update(sim=b, n=off)
        if do == "batch":
            s["out"] = torch.empty((off, 3), device="cuda")
        else:
            s["pins"] = np.concatenate(pins).astype(np.uint32)
            s["pos"] = np.concatenate(pos)
            s["host"] = [torch.empty((off, 3), pin_memory=True).numpy() for _ in range(case["frames"])]
        return s
    if do == "tree":
        g = np.random.default_rng(seed)
        body = _body(case["body"])
        s["xyz"], s["nrm"] = _poses(case, body.xyz, body.normals, case["poses"], g)
        nt = len(body.tris)
        s["tris"] = torch.from_numpy(body.tris.astype(np.int32)).cuda()
        s["outs"] = [[torch.zeros(n, dtype=torch.int32, device="cuda") for n in (nt, nt, max(nt - 1, 1), max(nt - 1, 1), 1)]
                     for _ in range(case["poses"])]
        return s
    if do == "fit":
        g = np.random.default_rng(seed)
        _, _, lists = _sheet(case["rows"], case["cols"])
        p = _params(case)
        x0 = _cloth_positions(case, g)
        ks = _stiffness(case, lists, p, g)
        lists = [scenes.SpringList(sl.row, sl.ent, k) for sl, k in zip(lists, ks)]
        body, bx = _body(case["body"]), _body_positions(case)
        s["sim"] = vs.Simulator(x0, lists, bx, body.tris, body.normals, params=p,
                                pinned=_pins(case["rows"], case["cols"]))
        s.update(x0=x0, zero=np.zeros_like(x0), target=_fit_target(x0, g))
        return s
    g, sim, p, x0, bx, body, faces = _single(case, seed)
    n = len(x0)
    s.update(sim=sim, n=n, out=torch.empty((n, 3), device="cuda"))
    if do == "drag":
        s["idx"], s["to"] = _targets(x0, case["rows"], case["cols"], g)
    if do == "body":
        s["poses"], s["pnrm"] = _poses(case, bx, body.normals, 64, g)
    if do == "output":
        sim.set_faces(faces)
        s["pos4"] = torch.empty((n, 4), device="cuda")
        s["vn"] = torch.empty((n, 3), device="cuda")
        s["fn"] = torch.empty((len(faces), 3), device="cuda")
    return s


def _fit_target(x0, g):
    """Where the fitted sheet should end: the sheet bent by a few centimetres."""
    a, b = g.uniform(2.0, 5.0, 2)
    y = 0.03 * np.sin(a * x0[:, 0].astype(np.float64)) * np.cos(b * x0[:, 2].astype(np.float64)) - 0.02
    return (x0 + np.stack([0.02 * x0[:, 0], y, -0.02 * x0[:, 2]], 1)).astype(np.float32)


# ---------------------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------------------
def run(s):
    do, case = s["do"], s["case"]
    if do == "drag":
        sim = s["sim"]
        sim.update_vertices(s["idx"], s["to"][s["k"] % 8])
        s["k"] += 1
        sim.simulate(case["steps"])
        sim.positions_device(_ptr(s["out"]))
        return s["out"]
    if do == "steps":
        s["sim"].simulate(case["steps"])
        s["sim"].positions_device(_ptr(s["out"]))
        return s["out"]
    if do == "body":
        sim = s["sim"]
        for _ in range(case["frames"]):
            k = s["k"] % 64
            s["k"] += 1
            sim.update_body_device(_ptr(s["poses"][k]), _ptr(s["pnrm"][k]))
            sim.simulate(case["steps"])
        sim.positions_device(_ptr(s["out"]))
        return s["out"]
    if do == "batch":
        s["sim"].step(case["steps"])
        s["sim"].positions_device(_ptr(s["out"]))
        return s["out"]
    if do == "stream":
        b = s["sim"]
        for f in range(case["frames"]):
            b.update_vertices(s["pins"], s["pos"])
            b.step(1)
            b.read_positions_async(s["host"][f])
            if f >= 2:
                b.wait_positions()
        for _ in range(min(2, case["frames"])):
            b.wait_positions()
        return s["host"]
    if do == "fit":
        sim = s["sim"]
        sim.set_state(s["x0"], s["x0"], s["zero"])
        sim.forward(case["steps"], case["every"])
        x = sim.positions()
        dk, ds = sim.backward((x - s["target"]) * np.float32(2.0 / len(x)))
        return dict(x=x, dk=dk, ds=ds)
    if do == "tree":
        L = vs.lib()
        for f, o in enumerate(s["outs"]):
            code = L.visg_lbvh_build_noalloc(_ptr(s["xyz"][f]), _ptr(s["nrm"][f]), s["xyz"].shape[1], _ptr(s["tris"]),
                                             len(s["tris"]), 0.003, 0.01, *[_ptr(t) for t in o],
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            if code:
                raise vs.VisgError(code, "tree")
        return s["outs"]
    sim = s["sim"]
    sim.simulate(case["steps"])
    if vs.lib().visg_render(sim.h, _ptr(s["pos4"]), _ptr(s["vn"]), _ptr(s["fn"]), 1, 1):
        raise RuntimeError("render")
    return [s["pos4"], s["vn"], s["fn"]]


# ---------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------
def _counts(case):
    """Vertices, directed springs, faces of the cloth; vertices, triangles of the body (by formula)."""
    r, c = case["rows"], case["cols"]
    n, f = r * c, 2 * (r - 1) * (c - 1)
    if r == c:
        e = 2 * (2 * r * (r - 1) + 2 * (r - 1) ** 2 + 2 * r * (r - 2))
    else:
        edges = r * (c - 1) + c * (r - 1) + (r - 1) * (c - 1)
        e = 2 * edges + 2 * (edges - 2 * (r + c - 2))
    return n, e, f


def work(case):
    """Inputs read once, outputs written once.  A step reads a vertex's x and x_old and its
    springs (end and rest length, 8 bytes) and writes x and x_old; what a run of steps
    leaves in between need not leave the chip and is not counted.  A spring takes about
    30 operations (45 damped, 150 for its derivative), a vertex about 40, a triangle of
    a tree about 200."""
    do = case["do"]
    per = 45 if case.get("physics") == "reference" else 30
    if do == "tree":
        b = _body(case["body"])
        nv, nt = len(b.xyz), len(b.tris)
        return dict(bytes=case["poses"] * (24 * nv + 12 * nt + 16 * nt), flops=case["poses"] * 200 * nt)
    if do in ("batch", "stream"):
        sides = np.random.default_rng(7).integers(case["lo"], case["hi"] + 1, case["garments"]).astype(np.int64)
        n = int((sides ** 2).sum())
        e = int((2 * (2 * sides * (sides - 1) + 2 * (sides - 1) ** 2 + 2 * sides * (sides - 2))).sum())
        if do == "batch":
            return dict(bytes=48 * n + 8 * e + 12 * n, flops=case["steps"] * (per * e + 40 * n))
        return dict(bytes=48 * n + 8 * e + 12 * n * case["frames"], flops=case["frames"] * (per * e + 40 * n))
    n, e, f = _counts(case)
    flops = case["steps"] * (per * e + 40 * n)
    moved = 48 * n + 8 * e
    if do == "fit":
        return dict(bytes=24 * n + 12 * e + 12 * n + 12 * n + 4 * e, flops=flops + case["steps"] * (per + 150) * e)
    if do == "body":
        b = _body(case["body"])
        nv, nt = len(b.xyz), len(b.tris)
        return dict(bytes=moved + 12 * n + case["frames"] * 24 * nv + 12 * nt,
                    flops=case["frames"] * (flops + 200 * nt))
    if do == "output":
        return dict(bytes=moved + 28 * n + 24 * f, flops=flops + 30 * f + 30 * n)
    return dict(bytes=moved + 12 * n, flops=flops)


# ---------------------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------------------
class _Step64:
    """The step in 64 bits for a sheet that does not reach its body: Verlet with damped springs."""

    def __init__(self, case, p, ks=None):
        _, _, lists = _sheet(case["rows"], case["cols"])
        self.p = p
        src, end, rest, k = [], [], [], []
        for l, sl in enumerate(lists):
            src.append(np.repeat(np.arange(len(sl.row) - 1), np.diff(sl.row.astype(np.int64))))
            end.append(sl.ent["end"].astype(np.int64))
            rest.append(sl.ent["rest"].astype(np.float64))
            k.append(np.full(len(sl.ent), p.list_k[l], np.float64) if ks is None else ks[l].astype(np.float64))

        def dev(a):
            return torch.from_numpy(np.concatenate(a)).cuda()

        self.src, self.end, self.rest, self.k = dev(src), dev(end), dev(rest), dev(k)
        n = case["rows"] * case["cols"]
        self.free = torch.ones((n, 1), dtype=torch.float64, device="cuda")
        self.free[torch.from_numpy(_pins(case["rows"], case["cols"]).astype(np.int64)).cuda()] = 0.0
        self.gravity = torch.tensor(list(p.gravity), dtype=torch.float64, device="cuda")

    def __call__(self, x, xo, k=None, gamma=None, damp=None, kd=None):
        p = self.p
        k = self.k if k is None else k
        gamma = p.verlet_damping if gamma is None else gamma
        damp = p.force_damping if damp is None else damp
        kd = p.spring_damping if kd is None else kd
        v = (x - xo) / p.dt
        d = x[self.src] - x[self.end] + 2.0 ** -23
        dv = v[self.src] - v[self.end]
        length = d.square().sum(1).sqrt()
        c = -k * (length - self.rest) + kd * (dv * d).sum(1) / length
        force = (self.gravity * p.mass + damp * v).index_add(0, self.src, (c / length)[:, None] * d)
        moved = x + gamma * (x - xo) + force / p.mass * p.dt * p.dt
        return self.free * moved + (1.0 - self.free) * x, x


def exact(case, seed):
    """Sheets that have not reached their body.  Where there is contact, the outputs hang
    on the float tests that choose each vertex's triangle, and have no 64-bit value; a
    tree's outputs are whole numbers."""
    do = case["do"]
    if do not in ("drag", "steps", "output", "fit") or case.get("settle") or case["gap"] < 0.1:
        return None
    if case["rows"] * case["cols"] * case["steps"] > 2_500_000:
        return None
    g = np.random.default_rng(seed)
    p = _params(case)
    x0 = _cloth_positions(case, g)
    x = torch.from_numpy(x0).cuda().double()
    xo = x.clone()
    if do == "fit":
        ks = _stiffness(case, _sheet(case["rows"], case["cols"])[2], p, g)
        target = torch.from_numpy(_fit_target(x0, g)).cuda().double()
        step = _Step64(case, p, ks)
        k = step.k.clone().requires_grad_()
        sc = [torch.tensor(float(v), dtype=torch.float64, device="cuda", requires_grad=True)
              for v in (p.verlet_damping, p.force_damping, p.spring_damping)]
        for _ in range(case["steps"]):
            x, xo = checkpoint(step, x, xo, k, *sc, use_reentrant=False)
        grads = torch.autograd.grad((x - target).square().sum() / len(x0), [k, *sc])
        return dict(x=x.detach().cpu().numpy(), dk=grads[0].cpu().numpy(),
                    ds=np.array([float(v) for v in grads[1:]]))
    step = _Step64(case, p)
    if do == "drag":
        idx, to = _targets(x0, case["rows"], case["cols"], g)
        at = torch.from_numpy(idx.astype(np.int64)).cuda()
        x[at] = torch.from_numpy(to[0]).cuda().double()
        xo[at] = x[at]
    for _ in range(case["steps"]):
        x, xo = step(x, xo)
    if do != "output":
        return x
    f = torch.from_numpy(_sheet(case["rows"], case["cols"])[1].astype(np.int64)).cuda()
    q = xo  # normals of the positions the last step started from
    fn = torch.linalg.cross(q[f[:, 1]] - q[f[:, 0]], q[f[:, 2]] - q[f[:, 0]])
    fn = fn / fn.norm(dim=1, keepdim=True)
    vn = torch.zeros_like(x)
    for j in range(3):
        vn = vn.index_add(0, f[:, j], fn)
    vn = vn / vn.norm(dim=1, keepdim=True)
    return [torch.cat([x, torch.ones_like(x[:, :1])], 1), vn, fn]
