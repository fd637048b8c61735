"""The elimination tree (tree_kernel.cuh, tree_host.h) against the oracle, on the CPU: the node
functions compiled for the host over a scalar type whose loads and stores are checked against the
levels they belong to, run through the program a launch follows, over the forms an instance can
take (simple and multiple edges, self-paired modes, loop weights, an unpaired vertex, batches; one
photon pair up to more nodes than a block holds) and several instances in one program."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = nat._nvcc()
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not available")
    path = str(tmp_path_factory.mktemp("tree") / "tree_check")
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "-o", path, os.path.join(HERE, "tree_check.cu")],
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert build.returncode == 0, build.stdout.decode()
    return path


def evaluate(exe, insts, budget, chip, split=False):
    words = [len(insts), budget, 4, chip]

    def put(x, count):
        x = np.zeros(count) if x is None else np.asarray(x).reshape(-1)
        for z in x.astype(complex):
            words.extend([repr(float(z.real)), repr(float(z.imag))])

    for inst in insts:
        s, n = inst.struct, inst.struct.n
        words += [s.kind, n, s.E, s.batch_max, s.cutoff, s.has_odd] + list(inst.reps)
        put(inst.A, n * n)
        put(inst.D, n)
        put(inst.oddV, n)
        words.extend([repr(s.oddloop[0]), repr(s.oddloop[1])])
    run = subprocess.run([exe] + ["split"] * split, input=" ".join(str(w) for w in words).encode(), stdout=subprocess.PIPE,
                         stderr=subprocess.STDOUT, timeout=120)
    assert run.returncode == 0, run.stdout.decode()
    v = np.array([[float(x) for x in line.split()] for line in run.stdout.decode().split("\n") if line])
    return v[:, 0] + 1j * v[:, 1]


def check(exe, inst, want):
    # the sums of these small instances cancel by less than 1e3, so 1e-11 leaves a factor of 100.
    # Whole levels; blocks of nodes; one coefficient a thread everywhere and tiles everywhere
    want = np.atleast_1d(np.asarray(want, dtype=complex))
    for budget, chip in ((1e9, 77824), (3e4, 64), (2e3, 32)):
        for split in (False, True):  # multiple edges as simple ones
            got = evaluate(exe, [inst], budget, chip, split)
            assert np.max(np.abs(got - want)) <= 1e-11 * np.max(np.abs(want)), (budget, chip, split, got, want)


@pytest.mark.parametrize("n", [2, 4, 6, 8, 10, 14, 18])
def test_simple_edges(exe, n):
    A = wl.complex_symmetric(n, seed=n)
    check(exe, tw.prepare_hafnian(A), complex(oracle.hafnian_repeated(A, [1] * n)))


@pytest.mark.parametrize("n", [2, 3, 4, 5, 9, 12, 15])
def test_loops(exe, n):
    A = wl.complex_symmetric(n, seed=40 + n)
    D = wl.complex_symmetric(n, seed=80 + n)[0]
    check(exe, tw.prepare_loop_hafnian(A, D, [1] * n), complex(oracle.hafnian_repeated(A, [1] * n, mu=D, loop=True)))


@pytest.mark.parametrize("reps", [[2], [6], [1, 1, 2], [2, 2], [4, 1, 1], [3, 3, 3, 1], [2, 2, 2, 2, 1, 1],
                                  [5, 1, 2, 2, 1, 1, 0, 2], [12, 10], [2] * 7, [3, 1, 1, 1, 2, 1, 1]])
@pytest.mark.parametrize("loop", [False, True])
def test_multiple_edges(exe, reps, loop):
    n = len(reps)
    A = wl.complex_symmetric(n, seed=sum(reps)) * 0.4
    D = wl.complex_symmetric(n, seed=7)[0]
    for extra in ([0, 1] if loop else [0]):  # one photon more: an unpaired vertex
        r = list(reps)
        r[0] += extra
        prep = tw.prepare_loop_hafnian(A, D, r) if loop else tw.prepare_hafnian(A, r)
        check(exe, prep, complex(oracle.hafnian_repeated(A, r, mu=D, loop=loop)))


@pytest.mark.parametrize("fixed", [[0, 0], [1, 0], [1, 1, 1, 1], [2, 1, 0, 2], [3, 1, 2], [1] * 7, [4, 4, 1]])
@pytest.mark.parametrize("cutoff", [1, 4, 7])
def test_batches(exe, fixed, cutoff):
    n = len(fixed) + 1
    A = wl.complex_symmetric(n, seed=n) * 0.5
    D = wl.complex_symmetric(n, seed=9)[0]
    want = [complex(oracle.hafnian_repeated(A, list(fixed) + [k], mu=D, loop=True)) if sum(fixed) + k else 1.0
            for k in range(cutoff + 1)]
    check(exe, tw.prepare_loop_hafnian_batch(A, D, list(fixed), cutoff), want)


def test_several_instances(exe):
    A, B = wl.complex_symmetric(9, seed=1), wl.complex_symmetric(12, seed=2)
    D = A[0] * 0.5
    insts = [tw.prepare_hafnian(B), tw.prepare_loop_hafnian(A, D, [1] * 9),
             tw.prepare_loop_hafnian_batch(A, D, [1, 0, 2, 1, 0, 1, 0, 0], 5),
             tw.prepare_loop_hafnian(A, D, [3, 1, 1, 2, 0, 1, 0, 1, 1]), tw.prepare_hafnian(B[:6, :6])]
    for budget, chip in ((1e9, 77824), (4e3, 64)):
        got = evaluate(exe, insts, budget, chip)
        want = np.concatenate([evaluate(exe, [i], 1e9, 77824) for i in insts])
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


def test_tree_macs():
    """The cost model's count against a walk over the levels by hand: n = 6, 3 edges, one step."""
    from thewalrus_gb300 import costmodel

    assert costmodel.tree_hafnian_macs(6) == 2 * 7 + 3 * 3  # entries of 4 vertices; three products to order 1
    assert costmodel.tree_hafnian_flops(40) == 6 * costmodel.tree_hafnian_macs(40) == 3 * costmodel.tree_hafnian_flops(40, False)
