"""The elimination tree's host estimates and sizes (tree_host.h) over every size an instance may have, on the CPU."""
import math
import os
import shutil
import subprocess

import pytest

from thewalrus_gb300 import _native as nat

HERE = os.path.dirname(os.path.abspath(__file__))
PLAIN, LOOP, LOOP_ODD = 0, 1, 2


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = nat._nvcc()
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not available")
    path = str(tmp_path_factory.mktemp("tree") / "tree_limits_check")
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "-o", path, os.path.join(HERE, "tree_limits_check.cu")],
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert build.returncode == 0, build.stdout.decode()
    return path


def estimates(exe, insts, walk=0, limit=1e18, node=24):
    words = [len(insts)]
    for kind, reps in insts:
        words += [kind, len(reps)] + list(reps)
    run = subprocess.run([exe, str(walk), str(limit), str(node)], input=" ".join(map(str, words)).encode(), stdout=subprocess.PIPE,
                         stderr=subprocess.STDOUT, timeout=60)
    assert run.returncode == 0, (run.returncode, run.stdout.decode())
    return [[float(x) for x in line.split()] for line in run.stdout.decode().split("\n") if line]


def test_work_is_the_walks(exe):
    insts = [(kind, reps) for kind in (PLAIN, LOOP, LOOP_ODD)
             for reps in ([1], [2], [3], [1] * 9, [2] * 6, [1, 2, 1, 3, 1], [2, 2, 1, 1, 1, 1, 1], [4, 3, 5])]
    for walk in (1e9, 2e3):
        for work, walked, _, _ in estimates(exe, insts, walk):
            assert abs(work - walked) <= 1e-12 * walked


@pytest.mark.parametrize("kind", [PLAIN, LOOP, LOOP_ODD])
@pytest.mark.parametrize("reps", [[2] * 21, [3] * 17, [1] + [2] * 21, [2] * 31, [3] * 21, [1] * 32, [7] * 9])
def test_levels_of_more_nodes_than_an_int_holds(exe, kind, reps):
    """Beyond 2^31 nodes in a level the estimate stays a number (it had divided by zero)."""
    (work, _, _, _), = estimates(exe, [(kind, reps)])
    # at least a multiply-add for every node before the last two edges; at most 12 products of 64 coefficients
    # and 32 lanes an entry, 2,279 entries a node, in levels that grow twofold to all the sign vectors
    least, most = math.prod(r + 1 for r in sorted(reps)[1:len(reps) - 2]), math.prod(r + 1 for r in reps)
    assert least < work < 2 * 12 * 2080 * 32 * 2279 * most


@pytest.mark.parametrize("node", [8, 16, 24, 32, 48])
def test_bytes_of_the_levels(exe, node):
    """A level takes its 200 MB or 64 nodes, whichever is more, and a tree no more than all of its levels and
    the scratch; within a limit that is refused or kept."""
    insts = [(kind, [r] * (k // r)) for kind in (PLAIN, LOOP, LOOP_ODD) for r in (1, 2, 3, 5, 9) for k in range(1, 64)
             if 0 < k // r <= 32]
    for (kind, reps), (_, _, fits, size) in zip(insts, estimates(exe, insts, node=node)):
        widest = 64 * 2279 * 64 * node  # 64 nodes of the most entries and coefficients
        assert fits and size <= (len(reps) + 3) * max(200e6, widest) + 1e6
        if kind == PLAIN and node == 24 and reps == [1] * 20:
            assert size < 1.4e9
    for limit in (1.5e9, 1e8, 1e6, 1):
        for _, _, fits, size in estimates(exe, insts, limit=limit, node=node):
            assert bool(fits) == (size <= limit)
