"""Trees where the choice of evaluation would take the terms: shapes whose terms are sooner, sums that keep
what they were, and multiple edges that would be taken as copies.  Every case says that a tree ran.

Tolerances: 1e-10 in FP64 and 1e-8 in double-float against the double-double terms, the bars of the other
tests; for the sums that cancel by 1e9, a hundred roundings of the terms' size."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "df": 1e-8, "dd": 4e-15}


def by_tree(inst, precision):
    plan = nat.Plan([inst], precision=precision + "-tree")
    assert plan.trees() == 1
    plan.execute()
    got = plan.read()
    plan.close()
    return got


def both(inst, precision):
    exact = precision.startswith("mod")
    got, want = by_tree(inst, precision), nat.run([inst], precision + "-terms" if exact else "dd-terms")
    if exact:
        assert np.array_equal(got, want)
    else:
        assert np.max(np.abs(got - want)) <= TOL[precision] * np.max(np.abs(want)), (got, want)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("reps", [[1], [2], [3], [4], [7], [3, 3], [8, 8], [2] * 6, [1, 1, 2], [1, 1, 1, 1, 2, 2, 3], [6, 5, 1, 1, 2],
                                  [9, 1, 4, 4], [3] * 6, [1, 2, 3, 4, 5], [3, 3, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1]])
def test_multiple_edges(reps, precision):
    """All the multiple edge phases, by their own recurrences: real and complex, loops, an unpaired vertex."""
    n = len(reps)
    A = wl.complex_symmetric(n, seed=sum(reps)) * 0.3
    D = wl.complex_symmetric(n, seed=3)[0] * 0.5
    for M, v in ((A, D), (np.abs(A), np.abs(D))):
        for r in (reps, [reps[0] + 1] + reps[1:]):
            if sum(r) % 2 == 0:
                both(tw.prepare_hafnian(M, r), precision)
            if sum(r) > 1:
                both(tw.prepare_loop_hafnian(M, v, r), precision)


@pytest.mark.parametrize("prime", [0, 4])
@pytest.mark.parametrize("reps", [[4], [3, 3], [2, 1, 3, 1, 1, 0, 2], [5, 4, 1], [2] * 5, [6, 2, 2, 1, 1]])
def test_multiple_edges_of_residues(reps, prime):
    n = len(reps)
    A = wl.adjacency01(n, seed=n, p=0.8) + np.diag(np.arange(float(n)))
    both(tw.prepare_loop_hafnian(A, np.arange(1.0, n + 1), reps), "mod%d" % prime)
    both(tw.prepare_loop_hafnian_batch(A, np.arange(1.0, n + 1), reps[:-1], 4), "mod%d" % prime)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("modes,cutoff,top", [(2, 3, 1), (3, 5, 4), (4, 6, 2), (6, 5, 3), (9, 8, 2)])
def test_batches(modes, cutoff, top, precision):
    for B, D, fixed, cut in wl.batch_loop_calls(count=3, seed=modes, modes=modes, cutoff=cutoff, max_fixed=top):
        # U D U^T is symmetric to rounding, which double-double does not call symmetric
        both(tw.prepare_loop_hafnian_batch((B + B.T) / 2, D, list(fixed), cut), precision)


@pytest.mark.parametrize("n", [23, 27, 30])
def test_double_float_loops(n):
    A = wl.complex_symmetric(n, seed=n)
    both(tw.prepare_loop_hafnian(A, A[0] * 0.7, None), "df")
    both(tw.prepare_loop_hafnian(A.real.copy(), A[0].real * 0.7, None), "df")


@pytest.mark.parametrize("precision", ["fp64", "df"])
@pytest.mark.parametrize("n", [18, 36, 38])
def test_signed_matrices(n, precision):
    """Sums of both signs cancel; the double-double tree is their value and is itself checked at n = 18."""
    inst = tw.prepare_hafnian(wl.real_signed(n, seed=n))
    want = by_tree(inst, "dd")
    if n < 20:
        both(inst, "dd")
    assert abs(by_tree(inst, precision)[0] - want[0]) <= TOL[precision] * abs(want[0])


@pytest.mark.parametrize("photons,max_rep", [(28, 3), (36, 2)])
def test_uncoupled_blocks(photons, max_rep):
    A, gamma, rpt = wl.gaussian_state_loop(modes=14, seed=2, photons=photons, max_rep=max_rep)
    inst = tw.prepare_loop_hafnian(A, gamma, list(rpt))
    want, mag = tw.run_with_magnitudes([inst], "dd")
    assert abs(by_tree(inst, "dd")[0] - want[0]) <= 4e-15 * abs(want[0])
    assert abs(by_tree(inst, "fp64")[0] - want[0]) <= 100 * 2.0 ** -53 * mag[0] + 1e-13 * abs(want[0])


@pytest.mark.parametrize("limit", [0, 1e6, 4e5])
def test_multiple_edges_in_blocks(limit):
    A = wl.complex_symmetric(8, seed=1) * 0.3
    D = A[0]
    for reps in ([3, 3, 2, 2, 1, 1, 1, 1], [4, 2, 2, 3, 2, 2, 1, 2]):
        inst = tw.prepare_loop_hafnian(A, D, reps)
        plan = nat.Plan([inst], precision="fp64-tree", max_workspace=limit)
        assert plan.trees() == 1
        plan.execute()
        want = nat.run([inst], "dd-terms")[0]
        assert abs(plan.read()[0] - want) <= 1e-10 * abs(want)


def test_the_routes_themselves():
    """What the choice takes by default, and that the two evaluations can be asked for."""
    plain = tw.prepare_hafnian(wl.complex_symmetric(24, seed=1))
    kept = [tw.prepare_hafnian(wl.real_signed(36, seed=1)), tw.prepare_loop_hafnian(*(lambda s: (s[0], s[1], list(s[2])))(
        wl.gaussian_state_loop(modes=14, seed=2, photons=28, max_rep=3)))]
    A = wl.complex_symmetric(8, seed=1)
    A[0, 1] *= 1 + 1e-6
    none = [plain.shard(1, 9), tw.prepare_hafnian(A), tw.prepare_hafnian(wl.complex_symmetric(8, seed=1), glynn=False)]
    assert nat.Plan([plain]).trees() == nat.Plan([plain], precision="fp64-tree").trees() == 1
    assert nat.Plan([plain], precision="fp64-terms").trees() == 0
    assert nat.Plan(kept).trees() == 0 and nat.Plan(kept, precision="fp64-tree").trees() == len(kept)
    assert nat.Plan(none).trees() == nat.Plan(none, precision="fp64-tree").trees() == 0
    assert nat.Plan([plain] + kept + none).trees() == 1
