"""A tree launch whose barrier gives up: with a single poll a CTA does not wait for the others, so that the
wait runs out at once.  The read is an error, the plan's next execution is not touched by it."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def instances(kind):
    if kind == "single":  # one launch, which reduces too
        return [tw.prepare_hafnian(wl.complex_symmetric(26, seed=1))]
    if kind == "types":  # launches of two scalar types, side by side
        return [tw.prepare_hafnian(wl.complex_symmetric(24, seed=1)), tw.prepare_hafnian(wl.real_nonneg(26, seed=1))]
    many = [tw.prepare_hafnian(wl.complex_symmetric(n, seed=n)) for n in (8, 12, 16, 20, 22, 24)] * 4
    return many + [many[0].shard(1, 5)]  # a per-term group and a reduction of their own


@pytest.mark.parametrize("kind", ["single", "types", "many"])
def test_a_wait_that_runs_out(kind):
    insts = instances(kind)
    plan = nat.Plan(insts)
    plan.execute()
    want = plan.read()
    for _ in range(2):
        nat.check(plan.lib.wg_plan_barrier_polls(plan.handle, 1))
        plan.execute()
        with pytest.raises(RuntimeError, match="gave up"):
            plan.read()
        nat.check(plan.lib.wg_plan_barrier_polls(plan.handle, 0))
        for _ in range(2):
            plan.execute()
            got = plan.read()
            assert np.all(np.abs(got - want) <= 1e-13 * np.abs(want))
