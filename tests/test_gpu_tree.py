"""The elimination tree on the GPU against the per-term sieve of the same precision, at the sizes
where its launches change: one task, a task queue, levels in one block and in several; tile
remainders (series of 1 to 20 coefficients); every scalar type; simple and multiple edges, loop
weights, an unpaired vertex, batches; mixed in one plan, replayed from a graph; matrices that are
not symmetric keep the per-term evaluation.

Tolerances: both sides are right to 1e-10 relative in FP64 (the bar of the other tests), 1e-8 in
double-float, to the last bits of complex128 in double-double and exactly in residues."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "df": 1e-8, "dd": 4e-15}


def close(got, want, precision):
    got, want = np.atleast_1d(got), np.atleast_1d(want)
    if precision.startswith("mod"):
        assert np.array_equal(got, want)
    else:
        assert np.max(np.abs(got - want)) <= TOL[precision] * np.max(np.abs(want)), (got, want)


def both(inst, precision):
    close(nat.run([inst], precision), nat.run([inst], precision + "-terms"), precision)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("n", [2, 4, 6, 8, 10, 16, 22, 24, 28])
def test_plain(n, precision):
    both(tw.prepare_hafnian(wl.complex_symmetric(n, seed=n)), precision)
    both(tw.prepare_hafnian(wl.real_nonneg(n, seed=n)), precision)


@pytest.mark.parametrize("n", [30, 32, 34, 36])
def test_plain_by_levels(n):
    both(tw.prepare_hafnian(wl.complex_symmetric(n, seed=n)), "fp64")
    both(tw.prepare_hafnian(wl.real_nonneg(n, seed=n)), "fp64")


@pytest.mark.parametrize("n", [6, 14, 24, 30])
def test_residues(n):
    inst = tw.prepare_hafnian(wl.adjacency01(n, seed=n, p=0.7))
    for k in range(5):
        both(inst, "mod%d" % k)
    A = wl.adjacency01(7, seed=n, p=0.7) + np.diag(np.arange(7.0))
    for reps in ([2, 1, 3, 1, 1, 0, 2], [1, 1, 2, 1, 2, 4, 2]):
        both(tw.prepare_loop_hafnian(A, np.arange(1.0, 8.0), reps), "mod1")
        both(tw.prepare_loop_hafnian_batch(A, np.arange(1.0, 8.0), reps[:6], 4), "mod2")


@pytest.mark.parametrize("copies", [1, 40])
@pytest.mark.parametrize("sizes", [(4,), (24,), (30, 12), (38,)])
@pytest.mark.parametrize("primes", [1, 2, 3, 5])
def test_primes_of_one_call(primes, sizes, copies):
    """Side by side, one after another (n = 38), beside per-term groups and with outputs for a
    reduction of their own."""
    insts = [tw.prepare_hafnian(wl.adjacency01(n, seed=n, p=0.6)) for n in sizes]
    if copies > 1:
        A = wl.adjacency01(6, seed=1, p=0.7) + np.diag(np.arange(6.0))
        insts += [tw.prepare_hafnian(wl.adjacency01(10, seed=3), glynn=False)]
        insts += [tw.prepare_loop_hafnian_batch(A, np.arange(1.0, 7.0), [2, 1, 3, 1, 1], 4)] * copies
    got = nat._run(insts, nat.WG_PREC_PRIMES + primes, 0, primes).real.reshape(primes, -1)
    for k in range(primes):
        assert np.array_equal(got[k], nat.run(insts, "mod%d-terms" % k).real)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("n", [3, 5, 8, 13, 20, 23, 27])
def test_loops(n, precision):
    A = wl.complex_symmetric(n, seed=n)
    both(tw.prepare_loop_hafnian(A, A[0] * 0.7, None), precision)
    both(tw.prepare_loop_hafnian(A.real.copy(), A[0].real * 0.7, None), precision)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("reps", [[4], [7], [3, 3], [2] * 6, [1, 1, 1, 1, 2, 2, 3], [6, 5, 1, 1, 2], [9, 1, 4, 4],
                                  [3, 3, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1], [1] * 12 + [3] * 4, [1] * 16 + [6, 6],
                                  [1] * 8 + [2] * 4 + [4] * 4, [1] * 12 + [5, 5, 9, 9]])
def test_multiple_edges(reps, precision):
    """FP64 against double-double terms: FP64 terms of many photons in one edge cancel by 10^5 and more."""
    def both(inst, precision):
        oracle = "dd" if precision == "fp64" else precision
        close(nat.run([inst], precision), nat.run([inst], oracle + "-terms"), precision)

    A = wl.complex_symmetric(len(reps), seed=sum(reps)) * 0.3
    D = wl.complex_symmetric(len(reps), seed=3)[0] * 0.5
    if sum(reps) % 2 == 0:
        both(tw.prepare_hafnian(A, reps), precision)
    both(tw.prepare_loop_hafnian(A, D, reps), precision)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("modes,cutoff,top", [(2, 3, 1), (4, 6, 2), (6, 5, 3), (9, 8, 2), (12, 6, 2)])
def test_batches(modes, cutoff, top, precision):
    for B, D, fixed, cut in wl.batch_loop_calls(count=2, seed=modes, modes=modes, cutoff=cutoff, max_fixed=top):
        both(tw.prepare_loop_hafnian_batch(B, D, list(fixed), cut), precision)


@pytest.mark.parametrize("fixed", [[3] * 4, [2] * 6, [1] * 8, [25, 25, 24, 24]])
def test_batches_of_any_shared_memory(fixed):
    """A CTA's shared memory grows with the outputs and the photon pairs: below, about and above the
    48 KB that a launch may use unasked, and (double-double) above what an SM has."""
    n = len(fixed) + 1
    A, D = wl.complex_symmetric(n, seed=n), wl.complex_symmetric(n, seed=5)[0] * 0.5
    for cutoff in range(1, 16):
        inst = tw.prepare_loop_hafnian_batch(A, D, fixed, cutoff)
        if max(fixed) < 10:
            both(inst, "fp64")
        both(inst, "dd")


@pytest.mark.parametrize("photons,max_rep", [(16, 4), (28, 3), (36, 2)])
def test_multiple_edges_by_levels(photons, max_rep):
    A, gamma, rpt = wl.gaussian_state_loop(modes=14, seed=2, photons=photons, max_rep=max_rep)
    inst = tw.prepare_loop_hafnian(A, gamma, list(rpt))
    # these sums cancel by up to 1e9: the double-double tree is the value, and FP64 keeps within a
    # hundred roundings of the terms' size
    want, mag = tw.run_with_magnitudes([inst], "dd")
    close(nat.run([inst], "dd"), want, "dd")
    assert abs(nat.run([inst], "fp64")[0] - want[0]) <= 100 * 2.0 ** -53 * mag[0] + 1e-13 * abs(want[0])


@pytest.mark.parametrize("options", [{}, {"use_graph": True}, {"serial_groups": True}])
def test_plan_of_every_kind(options):
    insts = [tw.prepare_hafnian(wl.complex_symmetric(n, seed=n)) for n in (8, 34, 20)]
    insts += [tw.prepare_hafnian(wl.real_nonneg(n, seed=n)) for n in (12, 26)]
    B, D, fixed, cut = wl.batch_loop_calls(count=1, seed=5, modes=8, cutoff=4)[0]
    insts.append(tw.prepare_loop_hafnian_batch(B, D, list(fixed), cut))
    insts.append(insts[0].shard(1, 7))  # a term range: per-term, in the same plan
    A = wl.complex_symmetric(10, seed=1)
    A[0, 1] *= 1 + 1e-6  # not symmetric to rounding: per-term as well
    insts.append(tw.prepare_hafnian(A))
    want = nat.run(insts, "fp64-terms")
    plan = nat.Plan(insts, **options)
    for _ in range(3):
        plan.execute()
        assert np.max(np.abs(plan.read() - want) / np.abs(want)) <= 1e-10
    # the per-term queries answer as a per-term plan does
    terms = nat.Plan(insts, precision="fp64-terms")
    terms.execute()
    assert np.array_equal(plan.read_magnitudes(), terms.read_magnitudes())
    a, b = plan.partials(), terms.partials()
    assert a[1] == b[1] and np.array_equal(a[0], b[0])


@pytest.mark.parametrize("n", [5, 6, 7, 9, 12, 21, 26])
def test_direct_route_is_the_general_one(n):
    """hafnian's single native call against the checks, pairing and preparation in Python: the same
    instance, so the same bits; complex, real, and complex with real values."""
    A = wl.complex_symmetric(n, seed=n)
    for M in (A, A.real.copy(), A.real.astype(complex)):
        for loop in ((False, True) if n % 2 == 0 else (True,)):
            prep = tw.prepare_loop_hafnian(M) if loop else tw.prepare_hafnian(M)
            assert tw.hafnian(M, loop=loop) == nat.run([prep])[0]
