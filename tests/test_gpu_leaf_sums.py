"""The leaves' sum of a tree: beyond a phase in FP64, for double-float too."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def test_double_float_leaves_are_added_in_fp64():
    """Non-negative matrices, whose leaves need 48 bits but for a few roundings: with the sum over them exact
    the results' error is below one rounding to 48 bits, 2^-49, root mean square over 60 matrices (1.55e-15;
    1.95e-15 with the leaves added in double-float, four levels of lanes and warps more)."""
    rel = []
    for seed in range(100, 160):
        inst = tw.prepare_hafnian(wl.real_nonneg(24, seed=seed))
        want = nat.run([inst], "dd")[0]
        rel.append(abs(nat.run([inst], "df")[0] - want) / abs(want))
    assert np.sqrt(np.mean(np.square(rel))) < 2.0 ** -49


@pytest.mark.parametrize("precision", ["fp64", "df", "dd"])
@pytest.mark.parametrize("limit", [0, 2e6, 3e5])
def test_sums_over_several_phases(precision, limit):
    """One instance whose leaves come in one phase and in up to hundreds: loops, an unpaired vertex, batches (a
    warp's outputs each in a lane) and multiple edges.  Against the per-term sum in double-double; 1e-8 and 1e-10
    are the bars of the other tests."""
    tol = {"fp64": 1e-10, "df": 1e-8, "dd": 1e-14}[precision]
    A = wl.complex_symmetric(17, seed=1) * 0.5
    D = A[0] * 0.7
    insts = [tw.prepare_hafnian(A[:16, :16]), tw.prepare_hafnian(np.abs(A[:16, :16])), tw.prepare_loop_hafnian(A, D, [1] * 17),
             tw.prepare_loop_hafnian(A[:8, :8], D[:8], [2, 3, 1, 1, 2, 1, 1, 2]),
             tw.prepare_loop_hafnian_batch(A[:9, :9], D[:9], [1, 2, 1, 2, 1, 0, 1, 2], 7),
             tw.prepare_loop_hafnian_batch(np.abs(A[:9, :9]), np.abs(D[:9]), [2, 2, 1, 1, 1, 1, 1, 1], 11)]
    for inst in insts:
        plan = nat.Plan([inst], precision=precision, max_workspace=limit)
        plan.execute()
        got, want = plan.read(), nat.run([inst], "dd-terms")
        assert np.all(np.abs(got - want) <= tol * np.max(np.abs(want)))
        plan.close()
