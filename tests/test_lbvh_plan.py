"""Where the bucket sort of a body tree keeps its keys.  A build that gives up at a bounded
wait leaves them behind, and the steps already queued still walk the tree: the slots
must not lie over its nodes or leaves, whose links and triangle numbers are followed
unchecked.  Trees that are only read out (the build without allocation) keep them in the
node array and must fit the static scratch."""
import os
import subprocess

import pytest

import simulator_gb300 as vs
from simulator_gb300._build import ARCH, LIBDIR, nvcc

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SIZES = (1, 2, 127, 128, 129, 1000, 19584, 32768, 262144, 262145, 524288, 524289, 1310720)
CAP, TARGET, MOST = 512, 128, 2048
SCRATCH = 9 << 20


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    vs.lib()  # the library is built
    exe = str(tmp_path_factory.mktemp("plan") / "lbvh_plan")
    r = subprocess.run([nvcc(), *ARCH, "-std=c++17", "-I", os.path.join(ROOT, "simulator_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), os.path.join(HERE, "lbvh_plan.cu"), "-o", exe, "-L", LIBDIR,
                        "-lvisgsim", "-Xlinker", f"-rpath={LIBDIR}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, *map(str, SIZES)], capture_output=True, text=True, check=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    return {(r[0], r[1]): r[2:] for r in rows}


@pytest.mark.parametrize("nt", SIZES)
def test_slots(layout, nt):
    total, buckets, slots, over = layout[nt, 1]
    assert buckets == (min(-(-nt // TARGET), MOST) if nt <= MOST * CAP // 2 else 0)
    assert slots >= 8 * CAP * buckets
    assert not over
    total, buckets, slots, _ = layout[nt, 0]
    assert slots == 0
    # in the node array: a bucket's slots up to the last triangle it can hold
    if buckets:
        assert 8 * (CAP * (buckets - 1) + min(CAP, nt)) <= 64 * max(nt - 1, 1)
    if nt <= 32768:
        assert total <= SCRATCH
