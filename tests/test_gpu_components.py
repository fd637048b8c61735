"""Real and imaginary part each to its own size.

A matrix X + i h Y of small h has an imaginary part h times a derivative (a nearly real state, a
derivative by a complex step), and one of purely imaginary entries a result with one part exactly
zero.  The per-term evaluation keeps both parts to their own relative accuracy, and so does the tree.

Tolerances are those of the other GPU tests (1e-10 in FP64, 1e-8 in double-float, to the last bits in
double-double), here on each component; X and Y are non-negative, so that neither part cancels."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "df": 1e-8, "dd": 4e-15}


def forms(n, h):
    """Instances of every kind over X + i h Y."""
    A = wl.real_nonneg(n, seed=n) + 1j * h * wl.real_nonneg(n, seed=n + 1)
    D = A[0] * 0.5
    yield tw.prepare_hafnian(A)
    yield tw.prepare_loop_hafnian(A, D, [1] * n)
    yield tw.prepare_loop_hafnian(A[:-1, :-1], D[:-1], [1] * (n - 1))
    m = n // 2
    reps = [2, 3] + [1] * (m - 2)
    yield tw.prepare_loop_hafnian(A[:m, :m], D[:m], reps)
    yield tw.prepare_loop_hafnian_batch(A[:m, :m], D[:m], reps[:m - 1], 4)


def close_by_component(got, want, precision):
    for g, w in ((got.real, want.real), (got.imag, want.imag)):
        assert np.all(np.abs(g - w) <= TOL[precision] * np.abs(w)), (precision, g, w)


@pytest.mark.parametrize("precision,h", [("fp64", 1.0), ("fp64", 1e-4), ("fp64", 1e-8), ("fp64", 1e-20), ("df", 1e-4),
                                         ("df", 1e-8), ("dd", 1e-8), ("dd", 1e-20)])
@pytest.mark.parametrize("n", [8, 12, 20])
def test_small_imaginary_parts(n, precision, h):
    for inst in forms(n, h):
        close_by_component(nat.run([inst], precision), nat.run([inst], "dd-terms"), precision)


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("n", [8, 14, 24])
def test_purely_imaginary_matrix(n, precision):
    X = wl.real_nonneg(n, seed=n)
    want = nat.run([tw.prepare_hafnian(X)], "dd-terms")[0].real
    got = nat.run([tw.prepare_hafnian(1j * X)], precision)[0] * (-1j) ** (n // 2)
    assert got.imag == 0 and abs(got.real - want) <= TOL[precision] * want


def test_small_parts_beside_others_in_one_plan():
    """One plan over matrices of both sorts, in any order."""
    n = 14
    near = [wl.real_nonneg(n, seed=s) * (1 + 0j) + 1e-12j * wl.real_nonneg(n, seed=s + 1) for s in (1, 4)]
    insts = [tw.prepare_hafnian(M) for M in (near[0], wl.complex_symmetric(18, seed=2), near[1], wl.real_nonneg(n, seed=9))]
    for precision in TOL:
        got, want = nat.run(insts, precision), nat.run(insts, "dd-terms")
        close_by_component(got[[0, 2]], want[[0, 2]], precision)
        assert np.all(np.abs(got - want) <= TOL[precision] * np.abs(want))


@pytest.mark.parametrize("pattern", [[1] * 10 + [0] * 4, [2, 1, 0, 3, 1, 1, 2, 0, 1, 1], [1, 2, 1, 1, 1, 1, 0, 2]])
def test_served_requests(pattern):
    """A resident state that is real but for parts of 1e-9: even and odd photon numbers."""
    A = wl.real_nonneg(16, seed=3) * 0.1 + 1e-10j * wl.real_nonneg(16, seed=4)
    gamma = A[0] * 3
    state = nat.DeviceState(A, gamma)
    for p in (pattern, pattern + [1]):
        p = p + [0] * (16 - len(p))
        plan = nat.Plan.from_requests(state, [tw.matched_reps(p)] * 2)
        plan.execute()
        close_by_component(plan.read(), nat.run([tw.prepare_loop_hafnian(A, gamma, p)] * 2, "dd-terms"), "fp64")


@pytest.mark.parametrize("h", [1e-4, 1e-9])
@pytest.mark.parametrize("fixed", [[1, 1], [1, 1, 1], [2, 1, 1], [2, 2, 1, 1, 1, 1]])
def test_batches_whose_mode_alone_is_complex(fixed, h):
    """Modes that are nearly real beside a batch mode of any phase: output 0 does not know the batch mode."""
    m = len(fixed) + 1
    A = wl.real_nonneg(m, seed=m) + 1j * h * wl.real_nonneg(m, seed=m + 1)
    D = A[0] * 0.5
    A[-1] = A[:, -1] = wl.complex_symmetric(m, seed=2)[0] * 3
    D[-1] = 2 + 1j
    inst = tw.prepare_loop_hafnian_batch(A, D, fixed, 4)
    for precision in ("fp64", "df", "dd"):
        got, want = nat.run([inst], precision), nat.run([inst], "dd-terms")
        close_by_component(got[:1], want[:1], precision)
        assert np.all(np.abs(got - want) <= TOL[precision] * np.abs(want))


@pytest.mark.parametrize("options", [{"use_graph": True}, {"serial_groups": True}, {"max_workspace": 3e6}])
def test_plan_of_both_nodes(options):
    """The launches of both sorts of nodes side by side, replayed from a graph, one after another, in blocks."""
    near = [wl.real_nonneg(n, seed=n) + 1e-9j * wl.real_nonneg(n, seed=n + 1) for n in (8, 20)]
    insts = [tw.prepare_hafnian(M) for M in (near[0], wl.complex_symmetric(22, seed=2), near[1], wl.real_nonneg(18, seed=9))]
    want = nat.run(insts, "dd-terms")
    plan = nat.Plan(insts, **options)
    assert plan.trees() == 4
    for _ in range(3):
        plan.execute()
        got = plan.read()
        close_by_component(got[[0, 2]], want[[0, 2]], "fp64")
        assert np.all(np.abs(got - want) <= TOL["fp64"] * np.abs(want))
